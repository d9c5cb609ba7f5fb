// smc_coop.cu -- kernels and launches of the cooperative SMC step (smc_coop.cuh).
#include <algorithm>
#include <atomic>
#include <cstring>
#include <memory>
#include <new>

#include "smc_coop.cuh"
#include "smc_coop_host.cuh"

namespace mckl_b200 {

using namespace coop;

namespace {

__device__ __forceinline__ Ctx make_ctx(Shared &sh, const Global &g, unsigned T)
{
    const bool cluster = T > 1 && T <= kMaxCluster;
    // no CTA stores into another's shared memory before that one runs
    if (cluster)
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    return Ctx{g, &sh, T, blockIdx.x, 0, 0, 0, 0, cluster};
}

// A tile's dynamic shared memory: its values and its 64-bit integers, padded.
template <int TILE>
struct TileMem {
    double v[padded(TILE)];
    long long q[padded(TILE)];
};

template <int THR, int PER>
__global__ void __launch_bounds__(THR, 1) k_coop_weight(Global g, unsigned T, uint64_t N, double *W,
    const double *v, int add_log, CoopResult *out)
{
    extern __shared__ __align__(16) unsigned char coop_dyn[];
    __shared__ Shared sh;
    TileMem<THR * PER> &tm = *reinterpret_cast<TileMem<THR * PER> *>(coop_dyn);
    Ctx c = make_ctx(sh, g, T);
    constexpr uint32_t TILE = THR * PER;
    const uint64_t base = static_cast<uint64_t>(c.tile) * TILE;
    double m = -__longlong_as_double(0x7ff0000000000000ll);
#pragma unroll 2
    for (int k = 0; k < PER; ++k) {
        const uint32_t o = k * THR + threadIdx.x;
        if (base + o < N) {
            const double lw = add_log ? __dadd_rn(dd::log(W[base + o]), v[base + o]) : v[base + o];
            tm.v[pad(o)] = lw;
            if (m < lw) m = lw;  // max_element: NaN never replaces (core/weight.hpp:184-196)
        }
    }
    WeightOut r;
    Approx ap;
    if (!weight_phase<THR, PER>(c, tm.v, tm.q, N, m, r, ap)) return;
    const double inv = __ddiv_rn(1.0, r.accw);
#pragma unroll 2
    for (int k = 0; k < PER; ++k) {
        const uint32_t o = k * THR + threadIdx.x;
        if (base + o < N) W[base + o] = __dmul_rn(inv, tm.v[pad(o)]);
    }
    if (c.tile == 0 && threadIdx.x == 0) {
        out->ess = r.ess;
        out->log_nc = __dadd_rn(r.lmax, dd::log(r.accw));
        out->accw = r.accw;
        out->lmax = r.lmax;
    }
}

template <int THR, int PER>
__global__ void __launch_bounds__(THR, 1) k_coop_resample(Global g, unsigned T, int scheme, uint64_t N,
    uint64_t M, const double *W, const double *canon, double *ubuf, uint64_t *rep, CoopResult *out)
{
    extern __shared__ __align__(16) unsigned char coop_dyn[];
    __shared__ Shared sh;
    TileMem<THR * PER> &tm = *reinterpret_cast<TileMem<THR * PER> *>(coop_dyn);
    Ctx c = make_ctx(sh, g, T);
    constexpr uint32_t TILE = THR * PER;
    const uint64_t base = static_cast<uint64_t>(c.tile) * TILE;
#pragma unroll 2
    for (int k = 0; k < PER; ++k) {
        const uint32_t o = k * THR + threadIdx.x;
        tm.v[pad(o)] = base + o < N ? W[base + o] : 0.0;
    }
    __syncthreads();
    uint64_t R;
    if (!resample_phase<THR, PER>(c, tm.v, tm.q, N, M, scheme, [canon](uint64_t j) { return __ldg(canon + j); },
            [W](uint64_t i) { return W[i]; }, ubuf, nullptr, &R, nullptr))
        return;
    __syncthreads();
#pragma unroll 2
    for (int k = 0; k < PER; ++k) {
        const uint32_t o = k * THR + threadIdx.x;
        if (base + o < N) rep[base + o] = static_cast<uint64_t>(tm.q[pad(o)]);
    }
    if (c.tile == 0 && threadIdx.x == 0) out->used = R;
}

template <int THR, int PER>
__global__ void __launch_bounds__(THR, 1) k_coop_index(Global g, unsigned T, uint64_t N, uint64_t M,
    const uint64_t *rep, uint32_t *surp, uint64_t *idx)
{
    extern __shared__ __align__(16) unsigned char coop_dyn[];
    __shared__ Shared sh;
    TileMem<THR * PER> &tm = *reinterpret_cast<TileMem<THR * PER> *>(coop_dyn);
    Ctx c = make_ctx(sh, g, T);
    constexpr uint32_t TILE = THR * PER;
    const uint64_t base = static_cast<uint64_t>(c.tile) * TILE;
#pragma unroll 2
    for (int k = 0; k < PER; ++k) {
        const uint32_t o = k * THR + threadIdx.x;
        tm.q[pad(o)] = base + o < N ? static_cast<long long>(rep[base + o]) : 0;
    }
    __syncthreads();
    index_phase<THR, PER>(c, tm.v, tm.q, N, M, surp, [idx](uint64_t d) { idx[d] = d; },
        [idx](uint64_t d, uint64_t p) { idx[d] = p; });
}

// ---------------------------------------------------------------------------
// The plain AR(1) filter: every step of SMCSampler's loop (pf.cu) in one
// kernel, the decision to resample taken by every CTA from the same ESS.
// Particles ping-pong between two buffers: a step reads its tile of one and
// writes the other, a resampling gathers inside the one just written (an empty
// slot from an occupied one), so a slow CTA's gather never meets the next
// step's writes.  Against the graph per step and its read-back: see pf.cu.
// ---------------------------------------------------------------------------
struct FilterArgs {
    uint64_t N, T;
    const double *y;  // device
    double phi, sx, sd0, lconst, hinv, equal, ess_limit;
    uint32_t mkey[2], rkey[2];
    int scheme;
    double *xb[2], *W;
    uint64_t *anc;
    double *ubuf, *ess;
    uint32_t *surp;
    uint8_t *resampled;
    unsigned long long *ties;
    double *loglik;
};

__device__ __noinline__ double log_rn(double x)
{
    return dd::log(x);
}

__device__ __noinline__ void sincos_accurate(double x, double *s, double *c)
{
    dd::sincos_dd(x, s, c);
}

__device__ __forceinline__ void sincos_rn(double x, double *s, double *c)
{
    if (!dd::sincos_quick(x, s, c)) {
        double a, b;
        sincos_accurate(x, &a, &b);
        *s = a;
        *c = b;
    }
}

// The Normal(0, sd) draws of step t for the tile's particles, normal_distribution's
// layout and arithmetic (rng.cu: k_normal, k_normal_odd), each handed to
// put(local particle, value).  The tile's words are staged in shared memory.
template <int THR, int PER, class Put>
__device__ __forceinline__ void tile_normals(Ctx &c, const PhiloxGen &g, uint64_t N, uint64_t t, double sd,
    const Put &put)
{
    constexpr uint32_t TILE = THR * PER;
    const uint64_t base = static_cast<uint64_t>(c.tile) * TILE;
    if (base >= N) return;
    const uint32_t len = static_cast<uint32_t>(min(static_cast<uint64_t>(TILE), N - base));
    const bool odd = (len & 1u) != 0;  // the tile of the last particle of an odd N
    const uint64_t a0 = t * (N + 2 * (N & 1)) + base, b0 = a0 >> 2;
    const uint32_t s0 = static_cast<uint32_t>(a0 & 3), nb = (s0 + len + (odd ? 2 : 0) + 3) >> 2;
    __syncthreads();  // the words share their memory with the windows
    for (uint32_t i = threadIdx.x; i < nb; i += THR) {
        uint32_t blk[4];
        g.block(Ctr{{b0 + i + 1, 0, 0, 0}}, blk);
        c.sh->words[i] = make_uint4(blk[0], blk[1], blk[2], blk[3]);
    }
    __syncthreads();
    const uint32_t *w = reinterpret_cast<const uint32_t *>(c.sh->words) + s0;
    const uint32_t full = len & ~1023u, nu = (len - full) / 2;  // pairs of the partial chunk
#pragma unroll 2
    for (uint32_t p = threadIdx.x; p < TILE / 2; p += THR) {
        const uint32_t cb = (p >> 9) * 1024, i = p & 511;
        const uint32_t half = cb < full ? 512 : nu;
        if (cb > full || (cb == full && i >= nu)) continue;
        double r = __dsqrt_rn(__dmul_rn(-2.0, log_rn(u01_f64(kOC, w[cb + i]))));
        double sn, cs;
        sincos_rn(__dmul_rn(RealOps<double>::kTwoPi, u01_f64(kOC, w[cb + half + i])), &sn, &cs);
        if (sd != 1.0) r = __dmul_rn(sd, r);
        put(cb + i, __dmul_rn(r, sn));
        put(cb + half + i, __dmul_rn(r, cs));
    }
    if (odd && threadIdx.x == THR - 1) {
        const double r = __dmul_rn(sd, __dsqrt_rn(__dmul_rn(-2.0, log_rn(u01_f64(kOC, w[len])))));
        double sn, cs;
        sincos_rn(__dmul_rn(RealOps<double>::kTwoPi, u01_f64(kOC, w[len + 1])), &sn, &cs);
        put(len - 1, __dadd_rn(0.0, __dmul_rn(r, cs)));
    }
}

template <int THR, int PER>
__global__ void __launch_bounds__(THR, 1) k_coop_filter(Global g, unsigned T, FilterArgs a)
{
    extern __shared__ __align__(16) unsigned char coop_dyn[];
    __shared__ Shared sh;
    TileMem<THR * PER> &tm = *reinterpret_cast<TileMem<THR * PER> *>(coop_dyn);
    Ctx c = make_ctx(sh, g, T);
    constexpr uint32_t TILE = THR * PER;
    const uint64_t N = a.N, base = static_cast<uint64_t>(c.tile) * TILE;
    const PhiloxGen gm{a.mkey[0], a.mkey[1]}, gr{a.rkey[0], a.rkey[1]};
    const bool lead = c.tile == 0 && threadIdx.x == 0;
    const double log_equal = log_rn(a.equal);
    double ll_sum = 0.0, ess = static_cast<double>(N), accw = 1.0;
    unsigned long long ties = 0;
    uint64_t rpos = 0;   // words of the resampling stream used so far
    bool flat = true;    // the weights are all equal
    int cur = 0;
    double *x = a.xb[0];
    Approx ap;           // of the step's terms
    tile_normals<THR, PER>(c, gm, N, 0, a.sd0, [&](uint32_t o, double e) { x[base + o] = e; });
    __syncthreads();
    for (uint64_t t = 0; t <= a.T; ++t) {
        if (t > 0) {
            const double yt = a.y[t], inv = __ddiv_rn(1.0, accw);
            double m = -__longlong_as_double(0x7ff0000000000000ll);
            double *xn = a.xb[cur ^ 1];
            // the normalised weights are 1 / accw times the terms kept in tm.v
            tile_normals<THR, PER>(c, gm, N, t, 1.0, [&](uint32_t o, double e) {
                const double v = __dadd_rn(__dmul_rn(a.phi, x[base + o]), __dmul_rn(a.sx, e));
                xn[base + o] = v;
                const double r = __dsub_rn(yt, v);
                const double ll = __dsub_rn(a.lconst, __dmul_rn(__dmul_rn(r, r), a.hinv));
                const double lw = __dadd_rn(flat ? log_equal : log_rn(__dmul_rn(inv, tm.v[pad(o)])), ll);
                tm.v[pad(o)] = lw;
                if (m < lw) m = lw;
            });
            cur ^= 1;
            x = xn;
            WeightOut r;
            if (!weight_phase<THR, PER>(c, tm.v, tm.q, N, m, r, ap)) return;
            accw = r.accw;
            ess = r.ess;
            flat = false;
            if (lead) ll_sum += __dadd_rn(r.lmax, log_rn(accw));
        }
        const bool res = ess < a.ess_limit;
        if (lead) {
            a.ess[t] = ess;
            a.resampled[t] = res ? 1 : 0;
        }
        if (!res) continue;
        // the weights themselves, for the folds (and for the residual schemes'
        // second look, in global memory)
        const double inv = __ddiv_rn(1.0, accw);
#pragma unroll 2
        for (int k = 0; k < PER; ++k) {
            const uint64_t i = base + threadIdx.x * PER + k;
            const double w = i < N ? (flat ? a.equal : __dmul_rn(inv, tm.v[at<PER>(k)])) : 0.0;
            tm.v[at<PER>(k)] = w;
            if ((a.scheme >= 3 || a.scheme == 0) && i < N) a.W[i] = w;
        }
        // the weights' approximate sums are the terms' times 1 / accw: a few
        // roundings more, which the classification's margin holds many times
        const Approx apw{__dmul_rn(inv, ap.A), __dmul_rn(inv, ap.own), __dmul_rn(inv, ap.M)};
        uint64_t R;
        const uint64_t rp = rpos;
        if (!resample_phase<THR, PER>(c, tm.v, tm.q, N, N, a.scheme,
                [&gr, rp](uint64_t j) {
                    const uint64_t w = rp + 2 * j;  // even: both words in one block
                    uint32_t blk[4];
                    gr.block(Ctr{{(w >> 2) + 1, 0, 0, 0}}, blk);
                    return (w & 2) ? u01_canonical2(blk[2], blk[3]) : u01_canonical2(blk[0], blk[1]);
                },
                [&a](uint64_t i) { return a.W[i]; }, a.ubuf, flat ? nullptr : &apw, &R, &ties))
            return;
        rpos += a.scheme % 3 == 2 ? 2 : 2 * R;
        __syncthreads();
        uint64_t *anc = a.anc ? a.anc + t * N : nullptr;
        if (!index_phase<THR, PER>(c, tm.v, tm.q, N, N, a.surp, [anc](uint64_t d) { if (anc) anc[d] = d; },
                [anc, x](uint64_t d, uint64_t p) {
                    if (anc) anc[d] = p;
                    x[d] = __ldcg(x + p);
                }))
            return;
        __syncthreads();
        flat = true;
        accw = 1.0;
    }
    // the final weights; the particles are in xb[cur], the caller's buffer
    const double inv = __ddiv_rn(1.0, accw);
#pragma unroll 2
    for (int k = 0; k < PER; ++k) {
        const uint32_t o = k * THR + threadIdx.x;
        if (base + o < N) a.W[base + o] = flat ? a.equal : __dmul_rn(inv, tm.v[pad(o)]);
    }
    if (ties) atomicAdd(a.ties, ties);
    if (lead) *a.loglik = ll_sum;
}

// ---------------------------------------------------------------------------
// launches
// ---------------------------------------------------------------------------
// scratch() slots: the results, and the working memory of each kind of call.  A
// launch's exchange slots are cleared before it, and all launches count epochs
// from 1, so between a call's clear and its launch no other may use the slots:
// two host threads that make different calls on one stream share none.
constexpr int kResultSlot = 9, kWeightSlot = 11, kResampleSlot = 12, kIndexSlot = 13, kFilterSlot = 14;
constexpr size_t kSlotBytes = (2 * kMaxVals + 1) * kMaxTiles * sizeof(ulonglong2);

// CTAs of `kernel` that the current device holds at once (0 when it cannot
// launch cooperatively); asked once per device.
template <class K>
int resident(K kernel, int threads, size_t dyn, std::atomic<int> *cache)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 16) return 0;
    int n = cache[dev].load(std::memory_order_relaxed);
    if (n) return n - 1;
    int sms = 0, coopl = 0, per_sm = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&coopl, cudaDevAttrCooperativeLaunch, dev);
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(dyn)) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, dyn) != cudaSuccess || !coopl) {
        cudaGetLastError();
        per_sm = 0;
    }
    n = std::min<int>(sms * per_sm, kMaxTiles);
    cache[dev].store(n + 1, std::memory_order_relaxed);
    return n;
}

// The tiling of n elements (see smc_coop.cuh).
struct Tiling {
    int threads, per;
    unsigned T;
};

Tiling tiling(uint64_t n)
{
    static constexpr int kShapes[][2] = {{512, 2}, {512, 4}, {1024, 3}, {1024, 4}, {1024, 5}, {1024, 6}, {1024, 7},
        {1024, 8}};
    for (const auto &k : kShapes) {
        const uint64_t tile = static_cast<uint64_t>(k[0]) * k[1], T = (n + tile - 1) / tile;
        if (T <= kMaxTiles) return {k[0], k[1], static_cast<unsigned>(T)};
    }
    return {0, 0, 0};
}

// Working memory (buffer `slot`) of a launch of T tiles over n elements with
// `extra` more bytes; the slots are cleared on the stream when there are exchanges.  The
// results have a small buffer of their own, zeroed when it is allocated: it never
// grows, so an error word that no call has read yet is kept.
int coop_scratch(int slot, const Tiling &t, uint64_t n, size_t extra, Global *g, CoopResult **res, char **more,
    cudaStream_t s)
{
    const size_t win = t.T > 1 ? align256(static_cast<size_t>(kWinSets) * t.T * kTileWin * sizeof(Window)) : 0;
    const size_t dots = align256((n + 1023) / 1024 * sizeof(double));
    *res = static_cast<CoopResult *>(scratch(kResultSlot, sizeof(CoopResult), s));
    char *p = static_cast<char *>(scratch(slot, align256(kSlotBytes) + win + dots + extra, s));
    if (!*res || !p) {
        set_error("scratch allocation failed");
        return MCKL_B200_ERR_NOMEM;
    }
    g->err = &(*res)->err;
    g->slots = reinterpret_cast<ulonglong2 *>(p);
    g->chain = g->slots + 2 * kMaxVals * kMaxTiles;
    if (t.T > 1) MB_CUDA(cudaMemsetAsync(p, 0, kSlotBytes, s));
    p += align256(kSlotBytes);
    g->win = reinterpret_cast<Window *>(p);
    p += win;
    g->dots = reinterpret_cast<double *>(p);
    *more = p + dots;
    return MCKL_B200_OK;
}

// Launch kernel instance K (T tiles) if the device holds it at once.
template <class K, class... Args>
int launch(K kernel, int threads, size_t dyn, std::atomic<int> *cache, unsigned T, cudaStream_t s, Args... args)
{
    if (static_cast<int>(T) > resident(kernel, threads, dyn, cache)) return kCoopNo;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(T);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = dyn;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    if (T <= kMaxCluster) {
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = T;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
    } else {
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
    }
    cfg.attrs = at;
    cfg.numAttrs = T > 1 ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, args...);
    if (e == cudaErrorCooperativeLaunchTooLarge) {  // fewer SMs than the device has (a partitioned context)
        cudaGetLastError();
        return kCoopNo;
    }
    MB_CUDA(e);
    count_launch();
    return MCKL_B200_OK;
}

#define COOP_SHAPE(KERNEL, THR, PER, SLOT, TILING, STREAM, ...) \
    if ((TILING).threads == THR && (TILING).per == PER)         \
        return launch(KERNEL<THR, PER>, THR, sizeof(TileMem<THR * PER>), cache_[SLOT], (TILING).T, STREAM, __VA_ARGS__);
#define COOP_LAUNCH(KERNEL, TILING, STREAM, ...)                          \
    [&]() -> int {                                                        \
        static std::atomic<int> cache_[8][16];                            \
        COOP_SHAPE(KERNEL, 512, 2, 0, TILING, STREAM, __VA_ARGS__)        \
        COOP_SHAPE(KERNEL, 512, 4, 1, TILING, STREAM, __VA_ARGS__)        \
        COOP_SHAPE(KERNEL, 1024, 3, 2, TILING, STREAM, __VA_ARGS__)       \
        COOP_SHAPE(KERNEL, 1024, 4, 3, TILING, STREAM, __VA_ARGS__)       \
        COOP_SHAPE(KERNEL, 1024, 5, 4, TILING, STREAM, __VA_ARGS__)       \
        COOP_SHAPE(KERNEL, 1024, 6, 5, TILING, STREAM, __VA_ARGS__)       \
        COOP_SHAPE(KERNEL, 1024, 7, 6, TILING, STREAM, __VA_ARGS__)       \
        COOP_SHAPE(KERNEL, 1024, 8, 7, TILING, STREAM, __VA_ARGS__)       \
        return kCoopNo;                                                   \
    }()

}  // namespace

bool coop_fits(uint64_t n)
{
    return tiling(n).T > 0;
}

int coop_weight(uint64_t N, double *W, const double *v, int add_log, CoopResult **res, cudaStream_t s)
{
    const Tiling t = tiling(N);
    if (!t.T) return kCoopNo;
    Global g;
    char *more;
    const int rc = coop_scratch(kWeightSlot, t, N, 0, &g, res, &more, s);
    if (rc != MCKL_B200_OK) return rc;
    return COOP_LAUNCH(k_coop_weight, t, s, g, t.T, N, W, v, add_log, *res);
}

int coop_resample(int scheme, uint64_t N, uint64_t M, const double *W, const double *canon, uint64_t *rep,
    CoopResult **res, cudaStream_t s)
{
    const uint64_t n = std::max<uint64_t>(std::max(N, M), 1);
    const Tiling t = tiling(n);
    if (!t.T) return kCoopNo;
    Global g;
    char *more;
    const int rc = coop_scratch(kResampleSlot, t, n, align256(n * sizeof(double)), &g, res, &more, s);
    if (rc != MCKL_B200_OK) return rc;
    return COOP_LAUNCH(k_coop_resample, t, s, g, t.T, scheme, N, M, W, canon, reinterpret_cast<double *>(more), rep,
        *res);
}

int coop_rep_to_index(uint64_t N, uint64_t M, const uint64_t *rep, uint64_t *idx, CoopResult **res, cudaStream_t s)
{
    const uint64_t n = std::max(N, M);
    const Tiling t = tiling(n);
    if (!t.T) return kCoopNo;
    Global g;
    char *more;
    const int rc = coop_scratch(kIndexSlot, t, n, align256(static_cast<size_t>(t.T) * t.threads * t.per * sizeof(uint32_t)),
        &g, res, &more, s);
    if (rc != MCKL_B200_OK) return rc;
    if (t.T == 1) *res = nullptr;
    return COOP_LAUNCH(k_coop_index, t, s, g, t.T, N, M, rep, reinterpret_cast<uint32_t *>(more), idx);
}

int coop_filter(const CoopFilter &f, double *loglik, double *ess, uint8_t *resampled, uint64_t *ties, cudaStream_t s)
{
    const uint64_t N = f.N, T = f.T;
    const Tiling t = tiling(N);
    if (!t.T) return kCoopNo;
    // results: loglik, ties, ess[T + 1], resampled[T + 1]
    const size_t rbytes = align256(16 + (T + 1) * 9);
    const size_t tile_words = static_cast<size_t>(t.T) * t.threads * t.per;
    Global g;
    CoopResult *res;
    char *p;
    int rc = coop_scratch(kFilterSlot, t, N,
        rbytes + align256((T + 1) * 8) + 2 * align256(N * 8) + align256(tile_words * 4), &g, &res, &p, s);
    if (rc != MCKL_B200_OK) return rc;
    auto take = [&p](size_t n) {
        char *q = p;
        p += align256(n);
        return q;
    };
    FilterArgs a{};
    char *rb = take(rbytes);
    a.loglik = reinterpret_cast<double *>(rb);
    a.ties = reinterpret_cast<unsigned long long *>(rb + 8);
    a.ess = reinterpret_cast<double *>(rb + 16);
    a.resampled = reinterpret_cast<uint8_t *>(rb + 16 + (T + 1) * 8);
    double *y = reinterpret_cast<double *>(take((T + 1) * 8));
    a.y = y;
    a.N = N;
    a.T = T;
    a.phi = f.phi;
    a.sx = f.sx;
    a.sd0 = f.sd0;
    a.lconst = f.lconst;
    a.hinv = f.hinv;
    a.equal = f.equal;
    a.ess_limit = f.ess_limit;
    for (int k = 0; k < 2; ++k) {
        a.mkey[k] = f.mkey[k];
        a.rkey[k] = f.rkey[k];
    }
    a.scheme = f.scheme;
    // the buffers change at each of the T steps: the particles end in f.x
    a.xb[T & 1] = f.x;
    a.xb[(T & 1) ^ 1] = reinterpret_cast<double *>(take(N * 8));
    a.W = f.W;
    a.anc = f.anc;
    a.ubuf = reinterpret_cast<double *>(take(N * 8));
    a.surp = reinterpret_cast<uint32_t *>(take(tile_words * 4));
    MB_CUDA(cudaMemcpyAsync(y, f.y, (T + 1) * 8, cudaMemcpyHostToDevice, s));
    MB_CUDA(cudaMemsetAsync(rb, 0, 16, s));
    rc = COOP_LAUNCH(k_coop_filter, t, s, g, t.T, a);
    if (rc != MCKL_B200_OK) return rc;
    std::unique_ptr<char[]> h(new (std::nothrow) char[rbytes]);
    if (!h) {
        set_error("particle filter: out of host memory");
        return MCKL_B200_ERR_NOMEM;
    }
    MB_CUDA(cudaMemcpyAsync(h.get(), rb, rbytes, cudaMemcpyDeviceToHost, s));
    CoopResult hr;
    rc = coop_read(res, &hr, s);
    if (rc != MCKL_B200_OK) return rc;
    const auto word = [&h](size_t off, auto v) {
        std::memcpy(&v, h.get() + off, sizeof(v));
        return v;
    };
    *loglik = word(0, 0.0);
    *ties = word(8, uint64_t{0});
    if (ess) std::memcpy(ess, h.get() + 16, (T + 1) * 8);
    if (resampled) std::memcpy(resampled, h.get() + 16 + (T + 1) * 8, T + 1);
    return MCKL_B200_OK;
}

int coop_read(CoopResult *res, CoopResult *host, cudaStream_t s)
{
    MB_CUDA(cudaMemcpyAsync(host, res, sizeof(CoopResult), cudaMemcpyDeviceToHost, s));
    MB_CUDA(cudaStreamSynchronize(s));
    if (host->err) {
        MB_CUDA(cudaMemsetAsync(res, 0, sizeof(int), s));
        set_error("cooperative SMC kernel: a wait exceeded its limit");
        return MCKL_B200_ERR_DEVICE;
    }
    return MCKL_B200_OK;
}

}  // namespace mckl_b200
