// pf_batched.cuh -- descriptors of the batched particle filter (pf_batched.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace mckl_b200 {

struct BatchedFilter {
    uint64_t n;         // particles
    uint64_t off;       // offset of this filter's particles in the work arrays
    double phi, sx, sd0, lconst, hinv, sy;
    // shadow run (FP64, follows the main run's decisions): its parameters
    double phi_s, sx_s, sd0_s, lconst_s, hinv_s;
    uint32_t mkey[2];   // model stream: Philox4x32 key
    uint32_t rkey[2];   // resampling stream: Philox4x32 key
};

struct BatchedArgs {
    BatchedFilter *filt;
    double *y;          // F x (T + 1) observations
    int T;
    double threshold;
    int fp64;           // 1: propagate in double, 0: in float
    void *xa, *xb, *lw; // particles (resampled in place; xb unused), log-weights
    uint32_t *scanS, *epos;
    double *loglik;
    uint32_t *nresampled;
    double *xsa = nullptr, *xsb = nullptr, *lws = nullptr;  // FP64 shadow (FP32 run only)
    double *loglik_shadow = nullptr;
    char *terms = nullptr;  // working memory of the filters run by clusters (null: none are):
                            // terms_clusters x joint_bytes(terms_units)
    uint64_t terms_units = 0;
    int terms_clusters = 0;
};

// Units of a filter of n particles with the entry of an odd last one, even.
inline uint64_t joint_units(uint64_t n)
{
    return (n / 1024 * 129 + n % 1024 / 2 + 2) / 2 * 2;
}

inline size_t joint_bytes(uint64_t units)
{
    return units * 40;  // two float4 and a double per unit
}

// sorted: the filters' particle counts, largest first (host).
int pf_batched_launch(const BatchedArgs &a, const int *order, const uint64_t *sorted, int nf, int threads,
    int ctas_per_sm, int *queue, cudaStream_t s);
// The first nj filters of the order by a cluster of kJointCtas CTAs each, the
// others by a CTA each (FP32, no shadow); share: the joint filters' part of the
// work, slots: CTAs the device holds.
constexpr int kJointCtas = 4;
constexpr uint64_t kJointMin = 4096;  // smaller filters stay on one CTA
int pf_batched_joint_launch(const BatchedArgs &a, const int *order, int nj, int nf, double share, int threads,
    int slots, int *queue, cudaStream_t s);

}  // namespace mckl_b200
