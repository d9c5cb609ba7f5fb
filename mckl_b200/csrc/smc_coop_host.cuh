// smc_coop_host.cuh -- host interface of the cooperative SMC step (smc_coop.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace mckl_b200 {

// Each of the calls below returns kCoopNo, having done nothing, when the cloud
// does not fit the chip at once (or cooperative launches are not possible);
// the caller then takes the multi-kernel path.
constexpr int kCoopNo = 1;

// Results of a call, in device memory of the stream's (CoopResult *res).
// err stays set until a call has reported it (coop_read): a wait that gave up in a
// call that does not synchronize is reported by the stream's next one that does.
struct CoopResult {
    int err, pad;
    double ess, log_nc, accw, lmax;
    uint64_t used;  // uniforms a resampling used
};

// Whether a cloud of n particles fits the chip at once.
bool coop_fits(uint64_t n);
// Weight::normalize of W (add_log: log W + v, else v).
int coop_weight(uint64_t N, double *W, const double *v, int add_log, CoopResult **res, cudaStream_t s);
// Replication counts; the uniforms of the engine's stream (canonical; one for
// the systematic schemes) are in `canon` (device).
int coop_resample(int scheme, uint64_t N, uint64_t M, const double *W, const double *canon, uint64_t *rep,
    CoopResult **res, cudaStream_t s);
// Parent indices from replication counts; *res is null when no wait could give up.
int coop_rep_to_index(uint64_t N, uint64_t M, const uint64_t *rep, uint64_t *idx, CoopResult **res, cudaStream_t s);
// The plain AR(1) particle filter (pf.cu), all of its steps in one kernel.
struct CoopFilter {
    uint64_t N, T;
    const double *y;  // host, T + 1
    double phi, sx, sd0, lconst, hinv, equal, ess_limit;
    uint32_t mkey[2], rkey[2];
    int scheme;
    double *x, *W;    // device, N
    uint64_t *anc;    // device, (T + 1) x N, or null
};
// Results on the host (synchronizes): ess and resampled hold T + 1 entries (nullable).
int coop_filter(const CoopFilter &f, double *loglik, double *ess, uint8_t *resampled, uint64_t *ties, cudaStream_t s);
// Copy a result to the host (synchronizes); an error when a wait gave up.
int coop_read(CoopResult *res, CoopResult *host, cudaStream_t s);

}  // namespace mckl_b200
