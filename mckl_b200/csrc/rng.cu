// rng.cu -- RNG fills and the U01 / Normal / Exponential transforms on sm_100a.
//
// Every kernel is a pure function of (generator key, first block counter,
// word offset): thread i of the grid computes its blocks straight from the
// counter, so there is no inter-thread dependency and no read traffic.  Three
// shapes cover every call:
//   * aligned: the stream starts on a block boundary and the output is
//     16-byte aligned -> each thread turns whole blocks into 128-bit stores,
//     the values of a last partial block in the same launch;
//   * shifted: many values (launch_words) from the middle of a block into a 16-byte
//     aligned output -> the same stores, the values shifted between lanes;
//   * staged: short calls and other alignments -> a CTA generates a tile of
//     blocks into shared memory and writes its outputs from there, coalesced.
// The Normal transform pairs the two halves of each 8192-byte chunk
// (random/normal_distribution.hpp:50-78), so one CTA owns one chunk and stages
// the chunk's words in shared memory.
#include <algorithm>
#include <atomic>
#include <type_traits>
#include <cstring>
#include <mutex>
#include <functional>
#include <map>

#include "common.cuh"
#include "dispatch.cuh"
#include "transforms.cuh"

namespace mckl_b200 {

// ---------------------------------------------------------------------------
// error state, scratch
// ---------------------------------------------------------------------------
static thread_local std::string g_last_error;
static std::atomic<uint64_t> g_launches{0};

void set_error(const std::string &msg)
{
    g_last_error = msg;
}

void count_launch()
{
    g_launches.fetch_add(1, std::memory_order_relaxed);
}

struct ScratchBuf {
    void *ptr = nullptr;
    size_t bytes = 0;
};

struct ScratchKey {
    int dev;
    cudaStream_t stream;
    int slot;
    bool operator<(const ScratchKey &o) const
    {
        if (dev != o.dev) return dev < o.dev;
        if (stream != o.stream) return std::less<cudaStream_t>()(stream, o.stream);
        return slot < o.slot;
    }
};

static std::mutex g_scratch_mu;
static std::map<ScratchKey, ScratchBuf> g_scratch;

// One buffer per (device, stream, slot): calls on different streams never
// share working memory, and calls on one stream are ordered by the stream.
// The buffers come from the stream-ordered allocator, so a buffer that must
// grow is released after the work already queued on its stream
// (cudaFreeAsync) and replaced on the same stream without synchronising the
// device.  Growing is refused while the stream is being captured (the
// allocation would belong to the graph).
void *scratch(int slot, size_t bytes, cudaStream_t stream)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
    std::lock_guard<std::mutex> lk(g_scratch_mu);
    ScratchBuf &b = g_scratch[ScratchKey{dev, stream, slot}];
    if (b.bytes < bytes) {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(stream, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) {
            set_error("working memory must grow during stream capture; make one call of this size on the "
                      "stream before capturing it");
            return nullptr;
        }
        if (b.ptr) {
            if (cudaFreeAsync(b.ptr, stream) != cudaSuccess) return nullptr;
            b.ptr = nullptr;
            b.bytes = 0;
        }
        const size_t want = std::max<size_t>(bytes, 1 << 20);
        if (cudaMallocAsync(&b.ptr, want, stream) != cudaSuccess) {
            b.ptr = nullptr;
            return nullptr;
        }
        // a new buffer's first bytes are zero (the cooperative kernels' error word)
        if (cudaMemsetAsync(b.ptr, 0, 256, stream) != cudaSuccess) {
            cudaFreeAsync(b.ptr, stream);
            b.ptr = nullptr;
            return nullptr;
        }
        b.bytes = want;
    }
    return b.ptr;
}

// Release every working buffer this library holds for `stream` on the
// current device (after the work queued on it).
int scratch_release(cudaStream_t stream)
{
    int dev = 0;
    MB_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(g_scratch_mu);
    for (auto it = g_scratch.begin(); it != g_scratch.end();) {
        if (it->first.dev == dev && it->first.stream == stream) {
            if (it->second.ptr) MB_CUDA(cudaFreeAsync(it->second.ptr, stream));
            it = g_scratch.erase(it);
        } else {
            ++it;
        }
    }
    return MCKL_B200_OK;
}

// ---------------------------------------------------------------------------
// launch geometry
// ---------------------------------------------------------------------------
static int sm_count()
{
    static int n = 0;
    if (n == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (n <= 0) n = 148;
    }
    return n;
}

static unsigned grid_for(uint64_t work_items, int threads, int ctas_per_sm)
{
    const uint64_t need = (work_items + threads - 1) / threads;
    const uint64_t cap = static_cast<uint64_t>(sm_count()) * ctas_per_sm;
    return static_cast<unsigned>(std::max<uint64_t>(1, std::min(need, cap)));
}

// ---------------------------------------------------------------------------
// device helpers
// ---------------------------------------------------------------------------
// Write block i into a shared staging buffer with 128-bit stores: consecutive
// lanes then fill consecutive 16-byte slots (no bank conflicts).
template <class G>
__device__ __forceinline__ void stage_block(uint32_t *st32, int i, const uint32_t (&blk)[G::kWords])
{
    uint4 *dst = reinterpret_cast<uint4 *>(st32) + i * (G::kWords / 4);
#pragma unroll
    for (int q = 0; q < G::kWords / 4; ++q) {
        dst[q] = make_uint4(blk[4 * q], blk[4 * q + 1], blk[4 * q + 2], blk[4 * q + 3]);
    }
}

// Store N values of R starting at a pointer known to be 16-byte aligned.
template <typename R, int N>
__device__ __forceinline__ void store_aligned(R *p, const R (&v)[N])
{
    if constexpr ((sizeof(R) * N) % 16 == 0) {
        constexpr int Q = static_cast<int>(sizeof(R) * N / 16);
        const uint4 *src = reinterpret_cast<const uint4 *>(v);
        uint4 *dst = reinterpret_cast<uint4 *>(p);
        // streaming stores: the output is written once and not read back here
#pragma unroll
        for (int q = 0; q < Q; ++q) __stcs(dst + q, src[q]);
    } else {
#pragma unroll
        for (int q = 0; q < N; ++q) p[q] = v[q];
    }
}

// ---------------------------------------------------------------------------
// Output functors: how words become outputs.
//   RawOut<W>        one word -> itself
//   U01Out<R,W>      one word -> U01 variant
//   Canon2Out        two u32 words -> canonical double
//   ExpOut<R,W>      one word -> log(U01OC) * (-1/lambda)
// ---------------------------------------------------------------------------
template <typename W>
struct RawOut {
    using out_t = W;
    static constexpr int kIn = 1;
    static constexpr bool kCheap = true;
    __device__ W operator()(const W *w) const { return w[0]; }
};

template <typename R, typename W>
struct U01Out {
    using out_t = R;
    static constexpr int kIn = 1;
    static constexpr bool kCheap = true;
    int variant;
    __device__ R operator()(const W *w) const { return RealOps<R>::u01(variant, w[0]); }
};

struct Canon2Out {
    using out_t = double;
    static constexpr int kIn = 2;
    static constexpr bool kCheap = true;
    __device__ double operator()(const uint32_t *w) const { return u01_canonical2(w[0], w[1]); }
};

template <typename R, typename W>
struct ExpOut {
    using out_t = R;
    static constexpr int kIn = 1;
    static constexpr bool kCheap = false;
    R a;  // -1 / lambda, rounded in R as the reference does
    __device__ R operator()(const W *w) const
    {
        const R u = RealOps<R>::u01(kOC, w[0]);
        return RealOps<R>::mul(a, RealOps<R>::log(u));
    }
};

// Outputs of 32 bytes per block, lane l of a warp holding block bw + l: each
// lane writing its own 32 bytes makes every 128-bit store instruction cover
// half of each sector it touches.  Instead instruction k writes chunk 32k + l
// of the warp's 1 KiB (half l % 2 of block 16k + l / 2, fetched by shuffles),
// so each store is contiguous across the warp.  Returns false, storing
// nothing, unless all 32 blocks of the warp exist (then every lane is here).
template <typename R, int N>
__device__ __forceinline__ bool store_warp32(R *out, uint64_t b, uint64_t nblk, const R (&v)[N])
{
    static_assert(sizeof(R) * N == 32, "32-byte blocks only");
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t bw = b - lane;  // block of lane 0
    if (bw + 31 >= nblk) return false;
    const uint4 c0 = reinterpret_cast<const uint4 *>(v)[0], c1 = reinterpret_cast<const uint4 *>(v)[1];
    uint4 *dst = reinterpret_cast<uint4 *>(out + bw * N);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int src = 16 * k + static_cast<int>(lane >> 1);
        uint4 a, h;
        a.x = __shfl_sync(0xffffffffu, c0.x, src);
        a.y = __shfl_sync(0xffffffffu, c0.y, src);
        a.z = __shfl_sync(0xffffffffu, c0.z, src);
        a.w = __shfl_sync(0xffffffffu, c0.w, src);
        h.x = __shfl_sync(0xffffffffu, c1.x, src);
        h.y = __shfl_sync(0xffffffffu, c1.y, src);
        h.z = __shfl_sync(0xffffffffu, c1.z, src);
        h.w = __shfl_sync(0xffffffffu, c1.w, src);
        __stcs(dst + 32 * k + lane, (lane & 1) ? h : a);
    }
    return true;
}

// The outputs of block b of a launch: a vector, or the first `rem` of the block
// after the last whole one.
template <typename R, int N>
__device__ __forceinline__ void store_block(R *out, uint64_t b, uint64_t nblk, uint32_t rem, const R (&v)[N])
{
    if (b < nblk) {
        store_aligned<R, N>(out + b * N, v);
    } else {
#pragma unroll
        for (int q = 0; q < N; ++q)
            if (q < static_cast<int>(rem)) out[b * N + q] = v[q];
    }
}

// Aligned shape: nblk whole blocks starting at counter `base`, and the first
// `rem` outputs of one more; block b feeds outputs [b * OPB, (b + 1) * OPB).
// `out` is 16-byte aligned.
template <class G, typename W, class F, int THREADS = 256, bool REM = true>
__global__ void __launch_bounds__(THREADS) k_blocks(G g, Ctr base, uint64_t nblk, uint32_t rem,
    typename F::out_t *out, F f)
{
    using R = typename F::out_t;
    constexpr int WPB = G::kWords / WordView<W>::kPer32;  // words per block
    constexpr int OPB = WPB / F::kIn;                     // outputs per block
    g.prepare();
    // four blocks per thread and iteration, a grid stride apart (each store
    // instruction stays coalesced across the warp): independent work to
    // overlap with the stores in flight; one for the transforms whose
    // per-value math (double-double log) needs the registers
    constexpr int U = F::kCheap ? 4 : 1;
    const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x, total = REM ? nblk + (rem ? 1 : 0) : nblk;
    for (uint64_t b0 = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; b0 < total; b0 += U * stride) {
#pragma unroll
        for (int i = 0; i < U; ++i) {
            const uint64_t b = b0 + i * stride;
            if (b >= total) break;
            uint32_t blk[G::kWords];
            g.block(ctr_add(base, b, G::kCtrWords), blk);
            W w[WPB];
#pragma unroll
            for (int j = 0; j < WPB; ++j) w[j] = WordView<W>::get(blk, j);
            R o[OPB];
#pragma unroll
            for (int j = 0; j < OPB; ++j) o[j] = f(w + j * F::kIn);
            // the shuffles pay only where the store, not the generator or the
            // transform, is the limit (Philox with a cheap transform)
            if constexpr (sizeof(R) * OPB == 32 && F::kCheap && std::is_same<G, PhiloxGen>::value) {
                if (store_warp32<R, OPB>(out, b, nblk, o)) continue;
            }
            if constexpr (REM) {
                store_block<R, OPB>(out, b, nblk, rem, o);
            } else {
                store_aligned<R, OPB>(out + b * OPB, o);
            }
        }
    }
}

// k_blocks for Philox launches whose block counters differ only in their low
// word (PhiloxLo: the counter-independent products folded once per launch).
template <typename W, class F, bool REM>
__global__ void __launch_bounds__(256) k_blocks_plo(PhiloxLo p, uint32_t nblk, uint32_t rem,
    typename F::out_t *out, F f)
{
    using R = typename F::out_t;
    constexpr int WPB = PhiloxGen::kWords / WordView<W>::kPer32;
    constexpr int OPB = WPB / F::kIn;
    const uint32_t stride = gridDim.x * blockDim.x, total = REM ? nblk + (rem ? 1 : 0) : nblk;
    const uint32_t first = blockIdx.x * blockDim.x + threadIdx.x;
    // 32-bit block numbers (total < 2^32): the loop's arithmetic is on the same
    // pipes as the generator's
    for (uint32_t b = first, left = first < total ? total - first : 0; left > 0;
         left = left > stride ? left - stride : 0, b += stride) {
        uint32_t blk[PhiloxGen::kWords];
        p.block(b, blk);
        W w[WPB];
#pragma unroll
        for (int j = 0; j < WPB; ++j) w[j] = WordView<W>::get(blk, j);
        R o[OPB];
#pragma unroll
        for (int j = 0; j < OPB; ++j) o[j] = f(w + j * F::kIn);
        if constexpr (sizeof(R) * OPB == 32 && F::kCheap) {
            if (store_warp32<R, OPB>(out, b, nblk, o)) continue;
        }
        if constexpr (REM) {
            store_block<R, OPB>(out, b, nblk, rem, o);
        } else {
            store_aligned<R, OPB>(out + static_cast<uint64_t>(b) * OPB, o);
        }
    }
}

// Shifted shape: outputs [0, ngroups OPB + rem) from a stream that starts at word
// `off` (not 0) of block `base`, one word per output, `out` 16-byte aligned.
// Every lane transforms a block of its own; the output group of OPB values at
// block b holds the block's values from `off` on and the first `off` of the next
// block, which the next lane has: the lanes shift their values down by powers
// of two with shuffles and store whole vectors.  A warp's last lane only serves
// the one before it (31 groups for 32 blocks).  Against the staged shape: no
// shared memory, no barriers, vector stores (5e6 single-precision Exponentials
// from ARS at an offset of one word: 31.0 -> 23.2 us).
template <class G, typename W, class F, int THREADS = 256>
__global__ void __launch_bounds__(THREADS) k_shifted(G g, Ctr base, uint32_t off, uint64_t ngroups,
    uint32_t rem, typename F::out_t *out, F f)
{
    using R = typename F::out_t;
    constexpr int WPB = G::kWords / WordView<W>::kPer32;
    g.prepare();
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t warps = static_cast<uint64_t>(gridDim.x) * (THREADS / 32), total = ngroups + (rem ? 1 : 0);
    for (uint64_t w = static_cast<uint64_t>(blockIdx.x) * (THREADS / 32) + threadIdx.x / 32; w * 31 < total;
         w += warps) {
        const uint64_t b = w * 31 + lane;  // block `total` serves the last group
        R o[WPB];
        if (b <= total) {
            uint32_t blk[G::kWords];
            g.block(ctr_add(base, b, G::kCtrWords), blk);
            W v[WPB];
#pragma unroll
            for (int j = 0; j < WPB; ++j) v[j] = WordView<W>::get(blk, j);
#pragma unroll
            for (int j = 0; j < WPB; ++j) o[j] = f(v + j);
        } else {
#pragma unroll
            for (int j = 0; j < WPB; ++j) o[j] = R(0);
        }
#pragma unroll
        for (int s = 1; s < WPB; s <<= 1) {
            if (off & s) {  // the same for every lane
                R t[WPB];
#pragma unroll
                for (int j = 0; j < s; ++j) t[j] = __shfl_down_sync(0xffffffffu, o[j], 1);
#pragma unroll
                for (int j = 0; j + s < WPB; ++j) o[j] = o[j + s];
#pragma unroll
                for (int j = 0; j < s; ++j) o[WPB - s + j] = t[j];
            }
        }
        if (lane < 31 && b < total) store_block<R, WPB>(out, b, ngroups, rem, o);
    }
}

// Staged shape: outputs [0, n) consume stream words off + kIn * [0, n) counted
// from word 0 of block `base`.  A CTA stages TB blocks per tile.
template <class G, typename W, class F, int TB>
__global__ void __launch_bounds__(256) k_staged(G g, Ctr base, uint32_t off, uint64_t n, typename F::out_t *out, F f)
{
    constexpr int WPB = G::kWords / WordView<W>::kPer32;
    constexpr int TW = TB * WPB;  // words per tile
    __shared__ __align__(16) uint32_t st32[TB * G::kWords];
    W *st = reinterpret_cast<W *>(st32);
    g.prepare();
    const uint64_t total = static_cast<uint64_t>(off) + n * F::kIn;  // stream words touched, from block start
    const uint64_t ntiles = (total + TW - 1) / TW;
    for (uint64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const uint64_t w0 = t * TW;
        for (int i = threadIdx.x; i < TB; i += blockDim.x) {
            if (w0 + static_cast<uint64_t>(i) * WPB < total) {
                uint32_t blk[G::kWords];
                g.block(ctr_add(base, t * TB + i, G::kCtrWords), blk);
                stage_block<G>(st32, i, blk);
            }
        }
        __syncthreads();
        // outputs whose first word lies in this tile; a 2-word output may
        // straddle into the next tile, which the last thread recomputes.
        for (int j = threadIdx.x; j < TW; j += blockDim.x) {
            const uint64_t s = w0 + j;  // stream word
            if (s < off || s >= total) continue;
            const uint64_t rel = s - off;
            if (rel % F::kIn != 0) continue;
            W w[F::kIn];
            bool ok = true;
#pragma unroll
            for (int q = 0; q < F::kIn; ++q) {
                if (j + q < TW) {
                    w[q] = st[j + q];
                } else {
                    ok = false;
                }
            }
            if (!ok) {
                // word j + 1 is in the next block: generate it directly
                const uint64_t s1 = s + 1;
                uint32_t blk[G::kWords];
                g.block(ctr_add(base, s1 / WPB, G::kCtrWords), blk);
                w[1] = WordView<W>::get(blk, static_cast<int>(s1 % WPB));
            }
            out[rel / F::kIn] = f(w);
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// Normal: one CTA per 8192-byte chunk.  Chunk c uses stream words
// [c K, c K + len) (relative to the call's first word), len = K or, for the last
// chunk of a call, what is left; word i < len / 2 is the radius uniform and word
// len / 2 + i the angle uniform of output pair (c K + i, c K + len / 2 + i).  An
// odd call's last value is mean + (sd sqrt(-2 log u)) cos(2 pi v), u and v the two
// words after the last chunk (random/normal_distribution.hpp:93-100).  All of a
// call is one launch.
//
// Double is bound by instruction issue and the FP64 pipe.  A pair fails the
// quick phases' rounding tests with probability about 0.008, so one warp
// iteration in five would take the accurate phases for one lane.  Such pairs are
// put on a list of the warp instead, and the list is worked off 32 at a time, at
// the latest when the warp has done its chunks.  CTAs of 128 threads (256 where
// the generator keeps a table per CTA) wait less at the two barriers of a chunk;
// calls of few chunks run 512 threads on each.
// 2^24 + 1 values (Threefry): 176.0 us before, 133.3 now (one CTA size
// of 256 threads and no list: 173.2).  Single precision has no list and a loop of its
// own: through the list's loop, with whole indices for every store, 2^24 values
// took 46.3 / 62.3 us (Philox / Threefry) against 44.2 / 60.0.
// ---------------------------------------------------------------------------
template <class G, typename W, typename R, int K, int THREADS>
__global__ void __launch_bounds__(THREADS) k_normal(G g, Ctr base, uint32_t off, uint64_t nchunks, uint32_t last_len,
    R *out, R mean, R sd)
{
    using O = RealOps<R>;
    constexpr bool kDefer = sizeof(R) == 8;
    constexpr int WPB = G::kWords / WordView<W>::kPer32;
    constexpr int NB = K / WPB + 1;  // blocks staged per chunk (one extra for misalignment or an odd call's two words)
    __shared__ __align__(16) uint32_t st32[NB * G::kWords];
    // per warp: pairs for the accurate phases, their first output's number with
    // len / 2 in the upper 16 bits, and their words
    __shared__ uint64_t l_at[kDefer ? THREADS / 32 : 1][kDefer ? 64 : 1];
    __shared__ W l_u[kDefer ? THREADS / 32 : 1][kDefer ? 64 : 1], l_v[kDefer ? THREADS / 32 : 1][kDefer ? 64 : 1];
    const W *st = reinterpret_cast<const W *>(st32);
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t cnt = 0;  // entries of the warp's list, below 32 between iterations
    g.prepare();
    auto put = [&](uint64_t i, uint64_t j, R lg, R sn, R cs) {
        R s = O::sqrt(O::mul(static_cast<R>(-2), lg));
        if (sd != static_cast<R>(1)) s = O::mul(sd, s);
        if (mean != static_cast<R>(0)) {
            out[i] = O::fma(s, sn, mean);
            out[j] = O::fma(s, cs, mean);
        } else {
            out[i] = O::mul(s, sn);
            out[j] = O::mul(s, cs);
        }
    };
    auto work_off = [&](uint32_t n) {  // the list's last n <= 32 entries
        if constexpr (kDefer) {
            __syncwarp();
            cnt -= n;
            if (lane < n) {
                const uint64_t at = l_at[warp][cnt + lane], i = at & 0xffffffffffffull;
                R lg, sn, cs;
                pair_accurate(O::u01(kOC, l_u[warp][cnt + lane]),
                    O::mul(O::kTwoPi, O::u01(kOC, l_v[warp][cnt + lane])), &lg, &sn, &cs);
                put(i, i + (at >> 48), lg, sn, cs);
            }
            __syncwarp();
        }
    };
    for (uint64_t c = blockIdx.x; c < nchunks; c += gridDim.x) {
        const uint32_t len = c + 1 == nchunks ? last_len : K, nu = len / 2;
        const bool odd = (len & 1u) != 0;
        const uint64_t a0 = static_cast<uint64_t>(off) + c * K;  // absolute word of the chunk start
        const uint64_t b0 = a0 / WPB;
        const uint32_t s0 = static_cast<uint32_t>(a0 % WPB);
        const int nb = static_cast<int>((s0 + len + (odd ? 2 : 0) + WPB - 1) / WPB);
        for (int i = threadIdx.x; i < nb; i += THREADS) {
            uint32_t blk[G::kWords];
            g.block(ctr_add(base, b0 + i, G::kCtrWords), blk);
            stage_block<G>(st32, i, blk);
        }
        __syncthreads();
        const uint64_t o = c * K;
        if constexpr (!kDefer) {
            R *oc = out + o;
            for (uint32_t p = threadIdx.x; p < nu; p += THREADS) {
                R s, sn, cs;
                pair_quick(O::u01(kOC, st[s0 + p]), O::mul(O::kTwoPi, O::u01(kOC, st[s0 + nu + p])), &s, &sn, &cs);
                s = O::sqrt(O::mul(static_cast<R>(-2), s));
                if (sd != static_cast<R>(1)) s = O::mul(sd, s);
                if (mean != static_cast<R>(0)) {
                    oc[p] = O::fma(s, sn, mean);
                    oc[nu + p] = O::fma(s, cs, mean);
                } else {
                    oc[p] = O::mul(s, sn);
                    oc[nu + p] = O::mul(s, cs);
                }
            }
        }
        for (uint32_t p0 = kDefer ? warp * 32 : nu; p0 < nu; p0 += THREADS) {
            const uint32_t p = p0 + lane;
            bool ok = true;
            if (p < nu) {
                R lg, sn, cs;
                ok = pair_quick(O::u01(kOC, st[s0 + p]), O::mul(O::kTwoPi, O::u01(kOC, st[s0 + nu + p])), &lg, &sn,
                    &cs);
                if (ok) put(o + p, o + nu + p, lg, sn, cs);
            }
            if constexpr (kDefer) {
                const uint32_t m = __ballot_sync(0xffffffffu, !ok);
                if (m) {
                    if (!ok) {
                        const uint32_t e = cnt + __popc(m & ((1u << lane) - 1u));
                        l_at[warp][e] = (o + p) | static_cast<uint64_t>(nu) << 48;
                        l_u[warp][e] = st[s0 + p];
                        l_v[warp][e] = st[s0 + nu + p];
                    }
                    cnt += __popc(m);
                    if (cnt >= 32) work_off(32);
                }
            }
        }
        if (odd && threadIdx.x == THREADS - 1) {
            const R a = O::sqrt(O::mul(static_cast<R>(-2), O::log(O::u01(kOC, st[s0 + len]))));
            const R cv = O::cos(O::mul(O::kTwoPi, O::u01(kOC, st[s0 + len + 1])));
            out[o + len - 1] = O::add(mean, O::mul(O::mul(sd, a), cv));
        }
        __syncthreads();
    }
    if (cnt) work_off(cnt);
}

// ---------------------------------------------------------------------------
// host dispatch
// ---------------------------------------------------------------------------
// Launch the word -> output transform F for n outputs from position (B, off).
template <class G, typename W, class F>
static int launch_words(const G &g, const Ctr &B, uint32_t off, uint64_t n, typename F::out_t *out,
    const F &f, cudaStream_t s)
{
    if (n == 0) return MCKL_B200_OK;
    constexpr int WPB = G::kWords / WordView<W>::kPer32;
    constexpr int OPB = WPB / F::kIn;
    // (a call of less than one block is staged: one to three double Exponentials of
    // Threefry 2.6 us on the device, 3.9 by a thread that transforms a whole block)
    const bool aligned = (off == 0) && n >= OPB && (reinterpret_cast<uintptr_t>(out) % 16 == 0);
    // ARS: 32 KiB of table per CTA bounds residency at 6 CTAs per SM
    const int ctas = std::is_same<G, ArsGen>::value ? 6 : 8;
    if (aligned) {
        const uint64_t nblk = n / OPB, total = (n + OPB - 1) / OPB;
        const uint32_t rem = static_cast<uint32_t>(n % OPB);
        if constexpr (std::is_same<G, PhiloxGen>::value) {
            // no carry out of the low counter word within this launch
            if ((B.w[0] & 0xffffffffull) + total <= 0xffffffffull) {
                // (the store of a partial block costs the whole fill 4 %)
                const PhiloxLo p = PhiloxLo::make(g, B);
                const unsigned grid = grid_for(total, 256, ctas);
                if (rem) {
                    k_blocks_plo<W, F, true><<<grid, 256, 0, s>>>(p, static_cast<uint32_t>(nblk), rem, out, f);
                } else {
                    k_blocks_plo<W, F, false><<<grid, 256, 0, s>>>(p, static_cast<uint32_t>(nblk), 0, out, f);
                }
                MB_LAUNCH_CHECK();
                return MCKL_B200_OK;
            }
        }
        if constexpr (std::is_same<G, ArsGen>::value) {
            // ARS with four round tables: one 1024-thread CTA per SM
            MB_CUDA(allow_dyn_smem(k_blocks<ArsGen4, W, F, 1024>, ArsGen4::kDynSmem));
            k_blocks<ArsGen4, W, F, 1024><<<grid_for(total, 1024, 1), 1024, ArsGen4::kDynSmem, s>>>(
                ArsGen4::from(g), B, nblk, rem, out, f);
        } else {
            MB_CUDA(allow_dyn_smem(k_blocks<G, W, F>, G::kDynSmem));
            k_blocks<G, W, F><<<grid_for(total, 256, ctas), 256, G::kDynSmem, s>>>(g, B, nblk, rem, out, f);
        }
        MB_LAUNCH_CHECK();
        return MCKL_B200_OK;
    }
    if constexpr (F::kIn == 1) {
        // Where the shifted shape is the faster one.  ARS sets up four tables per SM
        // for it, which pays once the staged shape has a third tile for an SM: words
        // (measured with a table set-up 0.5 us longer), staged / shifted, 30,000
        // blocks 3.8 / 4.7 us, 70,000 5.2 / 4.9, 75,776 6.2 / 4.9, 200,000 9.9 / 6.5;
        // double Exponentials 5.8 / 7.5, 6.8 / 7.6, 8.5 / 7.6, 12.6 / 11.3.  The
        // others from 4096 values: Philox words 1.8 / 1.5 us, 10^6 3.9 / 2.9; double
        // Exponentials 3.2 / 3.1, 7.6 / 7.3; Threefry's 4.8 / 4.6, 9.4 / 9.3 (500
        // values 3.1 / 4.4).
        const uint64_t ng = n / WPB;
        const bool enough =
            std::is_same<G, ArsGen>::value ? ng >= 2 * 256 * static_cast<uint64_t>(sm_count()) : n >= 4096;
        if (reinterpret_cast<uintptr_t>(out) % 16 == 0 && enough) {
            const uint64_t warps = (ng + 1 + 30) / 31;
            const uint32_t rem = static_cast<uint32_t>(n % WPB);
            if constexpr (std::is_same<G, ArsGen>::value) {
                MB_CUDA(allow_dyn_smem(k_shifted<ArsGen4, W, F, 1024>, ArsGen4::kDynSmem));
                k_shifted<ArsGen4, W, F, 1024><<<grid_for(warps * 32, 1024, 1), 1024, ArsGen4::kDynSmem, s>>>(
                    ArsGen4::from(g), B, off, ng, rem, out, f);
            } else {
                k_shifted<G, W, F><<<grid_for(warps * 32, 256, ctas), 256, 0, s>>>(g, B, off, ng, rem, out, f);
            }
            MB_LAUNCH_CHECK();
            return MCKL_B200_OK;
        }
    }
    const uint64_t tiles = (static_cast<uint64_t>(off) + n * F::kIn + 256 * WPB - 1) / (256 * WPB);
    MB_CUDA(allow_dyn_smem(k_staged<G, W, F, 256>, G::kDynSmem));
    k_staged<G, W, F, 256><<<grid_for(tiles * 256, 256, ctas), 256, G::kDynSmem, s>>>(g, B, off, n, out, f);
    MB_LAUNCH_CHECK();
    return MCKL_B200_OK;
}

static bool is64(uint32_t kind)
{
    return geom(kind).rbytes == 8;
}

// Engine calls made by the reference's BATCH_0 / BATCH_1 chunking
// (random/internal/common.hpp:89-122): n / K calls of K words (each followed
// by an empty call), then one call of n % K words.
static void advance_chunked(mckl_b200_engine_t &e, uint64_t n, uint64_t K, uint64_t words_per_out)
{
    advance_calls(e, n / K, K * words_per_out);
    advance_call(e, (n % K) * words_per_out);
}

template <typename R>
static int u01_impl(mckl_b200_engine_t *e, int variant, size_t n, R *r, void *stream)
{
    MB_CHECK_ARG(e != nullptr, "null engine");
    MB_CHECK_ARG(kind_valid(e->kind), "invalid engine kind");
    MB_CHECK_ARG(n == 0 || r != nullptr, "null output");
    Ctr B;
    uint32_t off;
    next_position(*e, B, off);
    cudaStream_t s = as_stream(stream);
    const bool canon2 = std::is_same<R, double>::value && variant == kCanonical && !is64(e->kind);
    int rc = with_generator(*e, [&](auto g) {
        using G = decltype(g);
        if (canon2) {
            return launch_words<G, uint32_t>(g, B, off, n, reinterpret_cast<double *>(r), Canon2Out{}, s);
        }
        if (is64(e->kind)) {
            return launch_words<G, uint64_t>(g, B, off, n, r, U01Out<R, uint64_t>{variant}, s);
        }
        return launch_words<G, uint32_t>(g, B, off, n, r, U01Out<R, uint32_t>{variant}, s);
    });
    if (rc != MCKL_B200_OK) return rc;
    advance_chunked(*e, n, 8192 / sizeof(R), canon2 ? 2 : 1);
    return MCKL_B200_OK;
}

template <typename R>
static int exponential_impl(mckl_b200_engine_t *e, size_t n, R *r, R lambda, void *stream)
{
    MB_CHECK_ARG(e != nullptr, "null engine");
    MB_CHECK_ARG(kind_valid(e->kind), "invalid engine kind");
    MB_CHECK_ARG(n == 0 || r != nullptr, "null output");
    MB_CHECK_ARG(lambda > 0, "lambda must be positive");
    Ctr B;
    uint32_t off;
    next_position(*e, B, off);
    cudaStream_t s = as_stream(stream);
    const R a = static_cast<R>(-1) / lambda;
    int rc = with_generator(*e, [&](auto g) {
        using G = decltype(g);
        if (is64(e->kind)) return launch_words<G, uint64_t>(g, B, off, n, r, ExpOut<R, uint64_t>{a}, s);
        return launch_words<G, uint32_t>(g, B, off, n, r, ExpOut<R, uint32_t>{a}, s);
    });
    if (rc != MCKL_B200_OK) return rc;
    advance_chunked(*e, n, 8192 / sizeof(R), 1);
    return MCKL_B200_OK;
}

template <typename R>
static int normal_impl(mckl_b200_engine_t *e, size_t n, R *r, R mean, R sd, void *stream)
{
    MB_CHECK_ARG(e != nullptr, "null engine");
    MB_CHECK_ARG(kind_valid(e->kind), "invalid engine kind");
    MB_CHECK_ARG(n == 0 || r != nullptr, "null output");
    MB_CHECK_ARG(sd > 0, "stddev must be positive");
    constexpr uint64_t K = 8192 / sizeof(R);
    Ctr B;
    uint32_t off;
    next_position(*e, B, off);
    cudaStream_t s = as_stream(stream);
    const uint64_t m = n / K, l = n % K;
    int rc = with_generator(*e, [&](auto g) {
        using G = decltype(g);
        auto run = [&](auto wtag) {
            using W = decltype(wtag);
            const uint64_t chunks = m + (l ? 1 : 0);
            if (!chunks) return static_cast<int>(MCKL_B200_OK);
            auto launch = [&](auto threads) {
                constexpr int T = decltype(threads)::value;
                MB_CUDA(allow_dyn_smem(k_normal<G, W, R, K, T>, G::kDynSmem));
                k_normal<G, W, R, K, T><<<grid_for(chunks * T, T, 2048 / T), T, G::kDynSmem, s>>>(g, B, off, chunks,
                    static_cast<uint32_t>(l ? l : K), r, mean, sd);
                MB_LAUNCH_CHECK();
                return static_cast<int>(MCKL_B200_OK);
            };
            // A chunk or two per SM: its latency counts, one pair per thread.  Device
            // time with 512 / 128 threads (ARS: 256), 148, 296 and 444 chunks, double:
            // Philox 5.5 / 6.5, 6.9 / 6.8, 9.0 / 7.8 us, Threefry 5.7 / 7.1, 7.3 / 7.3,
            // 11.1 / 7.9, ARS 7.4 / 7.7, 9.6 / 9.5, 12.2 / 11.7; single: Philox 2.6 /
            // 3.9, 3.4 / 4.2, 4.2 / 4.6.
            if (chunks <= 2 * static_cast<uint64_t>(sm_count())) return launch(std::integral_constant<int, 512>{});
            return launch(std::integral_constant<int, G::kDynSmem ? 256 : 128>{});
        };
        if (is64(e->kind)) return run(uint64_t{});
        return run(uint32_t{});
    });
    if (rc != MCKL_B200_OK) return rc;
    // engine calls: per chunk u01_oc(K) -> [K][0]; then u01_oc(l) -> [l];
    // odd n: two single-word draws
    advance_calls(*e, m, K);
    advance_call(*e, l);
    if (n % 2) {
        advance_call(*e, 1);
        advance_call(*e, 1);
    }
    return MCKL_B200_OK;
}

}  // namespace mckl_b200

using namespace mckl_b200;

extern "C" {

const char *mckl_b200_last_error(void)
{
    return g_last_error.c_str();
}

uint64_t mckl_b200_launch_count(void)
{
    return g_launches.load(std::memory_order_relaxed);
}

const char *mckl_b200_version(void)
{
    return "mckl_b200 0.2 (sm_100a)";
}

int mckl_b200_release_stream(void *stream)
{
    return scratch_release(as_stream(stream));
}

int mckl_b200_engine_seed(mckl_b200_engine_t *e, uint32_t kind, uint64_t seed)
{
    MB_CHECK_ARG(e != nullptr, "null engine");
    MB_CHECK_ARG(kind_valid(kind), "invalid engine kind");
    std::memset(e, 0, sizeof(*e));
    e->kind = kind;
    const bool k32 = (kind != MCKL_B200_THREEFRY4X64 && kind != MCKL_B200_THREEFRY4X64_64);
    e->key[0] = k32 ? (seed & 0xFFFFFFFFull) : seed;
    e->index = static_cast<uint32_t>(geom(kind).M);
    return MCKL_B200_OK;
}

int mckl_b200_engine_discard(mckl_b200_engine_t *e, uint64_t nskip)
{
    MB_CHECK_ARG(e != nullptr, "null engine");
    MB_CHECK_ARG(kind_valid(e->kind), "invalid engine kind");
    const Geom g = geom(e->kind);
    const uint64_t M = static_cast<uint64_t>(g.M);
    if (nskip == 0) return MCKL_B200_OK;
    const uint64_t idx = e->index < M ? e->index : M;
    const uint64_t remain = M - idx;
    if (nskip <= remain) {
        e->index = static_cast<uint32_t>(idx + nskip);
        return MCKL_B200_OK;
    }
    nskip -= remain;
    // increment(ctr, nskip / M * rate) with rate = 1 (result block == counter
    // size), including the reference's carry when ctr[0] == max - k
    // (random/internal/increment_generic.hpp:209-217), then one generated block.
    const uint64_t k = nskip / M;
    Ctr c = ctr_of(*e);
    if (c.w[0] < UINT64_MAX - k) {
        c.w[0] += k;
    } else {
        c.w[0] += k;
        for (int i = 1; i < g.cwords; ++i) {
            if (++c.w[i] != 0) break;
        }
    }
    c = ctr_add(c, 1, g.cwords);
    set_ctr(*e, c);
    e->index = static_cast<uint32_t>(nskip % M);
    return MCKL_B200_OK;
}

int mckl_b200_rand(mckl_b200_engine_t *e, size_t n, void *r, void *stream)
{
    MB_CHECK_ARG(e != nullptr, "null engine");
    MB_CHECK_ARG(kind_valid(e->kind), "invalid engine kind");
    MB_CHECK_ARG(n == 0 || r != nullptr, "null output");
    Ctr B;
    uint32_t off;
    next_position(*e, B, off);
    cudaStream_t s = as_stream(stream);
    int rc = with_generator(*e, [&](auto g) {
        using G = decltype(g);
        if (is64(e->kind)) {
            return launch_words<G, uint64_t>(g, B, off, n, static_cast<uint64_t *>(r), RawOut<uint64_t>{}, s);
        }
        return launch_words<G, uint32_t>(g, B, off, n, static_cast<uint32_t *>(r), RawOut<uint32_t>{}, s);
    });
    if (rc != MCKL_B200_OK) return rc;
    advance_call(*e, n);
    return MCKL_B200_OK;
}

int mckl_b200_philox4x32_kernel(uint64_t ctr[2], size_t n, void *r, const uint32_t key[2], void *stream)
{
    MB_CHECK_ARG(ctr != nullptr && key != nullptr, "null ctr/key");
    MB_CHECK_ARG(n == 0 || r != nullptr, "null output");
    Ctr B{{ctr[0], ctr[1], 0, 0}};
    B = ctr_add(B, 1, 2);
    PhiloxGen g{key[0], key[1]};
    int rc = launch_words<PhiloxGen, uint32_t>(g, B, 0, n * 4, static_cast<uint32_t *>(r), RawOut<uint32_t>{},
        as_stream(stream));
    if (rc != MCKL_B200_OK) return rc;
    Ctr E = ctr_add(Ctr{{ctr[0], ctr[1], 0, 0}}, n, 2);
    ctr[0] = E.w[0];
    ctr[1] = E.w[1];
    return MCKL_B200_OK;
}

int mckl_b200_threefry4x64_kernel(uint64_t ctr[4], size_t n, void *r, const uint64_t key[4],
    const uint64_t tweak[2], void *stream)
{
    MB_CHECK_ARG(ctr != nullptr && key != nullptr, "null ctr/key");
    MB_CHECK_ARG(n == 0 || r != nullptr, "null output");
    const uint64_t zero[2] = {0, 0};
    ThreefryGen g = ThreefryGen::make(key, tweak ? tweak : zero);
    Ctr C{{ctr[0], ctr[1], ctr[2], ctr[3]}};
    int rc = launch_words<ThreefryGen, uint32_t>(g, ctr_add(C, 1, 4), 0, n * 8, static_cast<uint32_t *>(r),
        RawOut<uint32_t>{}, as_stream(stream));
    if (rc != MCKL_B200_OK) return rc;
    Ctr E = ctr_add(C, n, 4);
    for (int i = 0; i < 4; ++i) ctr[i] = E.w[i];
    return MCKL_B200_OK;
}

int mckl_b200_ars_kernel(uint64_t ctr[2], size_t n, void *r, const uint32_t key[4], void *stream)
{
    MB_CHECK_ARG(ctr != nullptr && key != nullptr, "null ctr/key");
    MB_CHECK_ARG(n == 0 || r != nullptr, "null output");
    const uint64_t k64[4] = {key[0], key[1], key[2], key[3]};
    ArsGen g = ArsGen::make(k64);
    Ctr C{{ctr[0], ctr[1], 0, 0}};
    int rc = launch_words<ArsGen, uint32_t>(g, ctr_add(C, 1, 2), 0, n * 4, static_cast<uint32_t *>(r),
        RawOut<uint32_t>{}, as_stream(stream));
    if (rc != MCKL_B200_OK) return rc;
    Ctr E = ctr_add(C, n, 2);
    ctr[0] = E.w[0];
    ctr[1] = E.w[1];
    return MCKL_B200_OK;
}

#define MB_U01(name, variant)                                                                      \
    int mckl_b200_u01_##name##_f32(mckl_b200_engine_t *e, size_t n, float *r, void *stream)          \
    {                                                                                              \
        return u01_impl<float>(e, variant, n, r, stream);                                          \
    }                                                                                              \
    int mckl_b200_u01_##name##_f64(mckl_b200_engine_t *e, size_t n, double *r, void *stream)         \
    {                                                                                              \
        return u01_impl<double>(e, variant, n, r, stream);                                         \
    }

MB_U01(canonical, kCanonical)
MB_U01(cc, kCC)
MB_U01(co, kCO)
MB_U01(oc, kOC)
MB_U01(oo, kOO)

int mckl_b200_normal_f32(mckl_b200_engine_t *e, size_t n, float *r, float mean, float sd, void *stream)
{
    return normal_impl<float>(e, n, r, mean, sd, stream);
}

int mckl_b200_normal_f64(mckl_b200_engine_t *e, size_t n, double *r, double mean, double sd, void *stream)
{
    return normal_impl<double>(e, n, r, mean, sd, stream);
}

int mckl_b200_exponential_f32(mckl_b200_engine_t *e, size_t n, float *r, float lambda, void *stream)
{
    return exponential_impl<float>(e, n, r, lambda, stream);
}

int mckl_b200_exponential_f64(mckl_b200_engine_t *e, size_t n, double *r, double lambda, void *stream)
{
    return exponential_impl<double>(e, n, r, lambda, stream);
}

}  // extern "C"
