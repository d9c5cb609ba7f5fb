// pf_batched_joint.cu -- launches of the batched filters whose largest are run
// by a cluster of CTAs each (k_pf_batched_joint, pf_batched_kernel.cuh).
#include <algorithm>

#include "pf_batched_kernel.cuh"

namespace mckl_b200 {

using namespace batched_detail;

namespace {

template <int THREADS>
int joint_one(const BatchedArgs &a, const int *order, int nj, int nf, double share, int slots, int *queue,
    cudaStream_t s)
{
    constexpr int C = kJointCtas;
    const uint64_t want = static_cast<uint64_t>(nj) * C + (nf - nj + C - 1) / C * C;
    const int clusters = std::max(1, static_cast<int>(std::min<uint64_t>(want, slots)) / C);
    const int nct = std::min(clusters, a.terms_clusters);
    // clusters that start with the joint filters: one each when there is room
    // for everything at once, else their share of the work
    const int room = nj + (nf - nj + C - 1) / C;
    const int ncj = std::max(1, std::min(nct, room <= clusters ? nj : static_cast<int>(share * clusters + 0.5)));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(clusters * C);
    cfg.blockDim = dim3(THREADS);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = C;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    MB_CUDA(cudaMemsetAsync(queue, 0, 2 * sizeof(int), s));
    MB_CUDA(cudaLaunchKernelEx(&cfg, k_pf_batched_joint<float, THREADS, 1024 / THREADS, C>,
        static_cast<const BatchedFilter *>(a.filt), order, nj, nf, ncj, nct, static_cast<const double *>(a.y), a.T,
        a.threshold, static_cast<float *>(a.xa), static_cast<float *>(a.lw), a.scanS, a.epos, a.loglik, a.nresampled,
        queue, a.terms, a.terms_units));
    count_launch();
    return MCKL_B200_OK;
}

}  // namespace

int pf_batched_joint_launch(const BatchedArgs &a, const int *order, int nj, int nf, double share, int threads,
    int slots, int *queue, cudaStream_t s)
{
    switch (threads) {
        case 128: return joint_one<128>(a, order, nj, nf, share, slots, queue, s);
        case 256: return joint_one<256>(a, order, nj, nf, share, slots, queue, s);
        case 512: return joint_one<512>(a, order, nj, nf, share, slots, queue, s);
        default: return joint_one<1024>(a, order, nj, nf, share, slots, queue, s);
    }
}

}  // namespace mckl_b200
