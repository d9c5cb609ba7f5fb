// fold_classify.cuh -- which elements of a sequential fold are certain integer
// steps (fold.cuh), shared by the multi-kernel fold (fold.cu) and the
// cooperative SMC kernels (smc_coop.cuh).
#pragma once

#include "fold.cuh"

namespace mckl_b200 {

__device__ __forceinline__ double ulp_of(double v)
{
    const int eb = biased_exp(v);
    return grid_unit(eb);
}

// ---------------------------------------------------------------------------
// Approximate partial sums and the classification of every element.
//
// A_j is a parallel (tree) sum of s0 + x_0 + ... + x_j; S_j the sequential
// fold.  Both are sums of nonnegative terms, so |A_j - S_j| <= (j + 1 + D)
// 2^-53 A_j (first order) with D the depth of A's summation tree (below
// 100 + T / 1024 here: 8 sequential adds per thread, two CTA scans, the
// tile scan with its carries).  ulp(A) > 2^-53 A, so a margin of
// 2 (j + 1) + 2 T + 160 ulps of A_j holds S_j with room to spare: when
// [A_j - margin, A_j + margin] lies inside one binade, S_j certainly does.
// ---------------------------------------------------------------------------
//
// Below 2^-1021 (biased exponent 0 or 1) every sum is exact: all partial
// sums of nonnegative terms are at most the total, and any sum of multiples
// of 2^-1074 below 2^-1021 is representable.  A tree sum below 2^-1021 is
// therefore the exact sum, which the sequential fold also reaches, and its
// binade is certain (this includes zero sums).
//
// The sequential fold never decreases and rounds monotonically, so S_j is at
// least the largest term so far, M_j: the lower end is max(A - margin, M_j).
// Where one term dominates -- degenerate weights, whose largest term is
// exactly 1 = 2^0 with a tiny remainder -- the sum sits just above a binade
// boundary that the margin alone would straddle.
__device__ __forceinline__ int certain_binade(double A, uint64_t j, uint64_t T, double M)
{
    if (biased_exp(A) <= 1 && A >= 0.0) return biased_exp(A);
    const double m = (2.0 * static_cast<double>(j + 1) + 2.0 * static_cast<double>(T) + 160.0) * ulp_of(A);
    const double lo = fmax(__dsub_rn(A, m), M), hi = __dadd_rn(A, m);
    if (!(lo > 0.0)) return -1;
    const int e = biased_exp(lo);
    if (e == 0x7ff || biased_exp(hi) != e) return -1;
    return e;
}

// Element j = i0 + k is a RUN element when the binades of S_{j-1} and S_j
// are certain and equal and x_j's grid increment at that binade has no event
// (tie, too large): then S_j = S_{j-1} + u q_j exactly.  Every other element
// is a WINDOW: the walk folds it with a real double add.  Returns, per
// element, q (0 for windows), the window bit and the certain binade of
// S_{j-1} (-1: uncertain).
//
// Fast case: S_{i0-1} .. S_{i0+PER-1} all lie in [A_before - m, A_end + m]
// (the partial sums grow, and A_end = A_before + the thread's own sum is a
// summation tree of the same depth as the per-element A_j), with m the margin
// of the last element, the largest.  When that interval lies in one binade,
// every element's binade is certain and the same, and only its increment
// remains to be checked.
template <int PER>
__device__ __forceinline__ void classify(const double (&xv)[PER], uint64_t i0, uint64_t n, uint64_t T, double s0,
    double Abefore, double own, double Mbefore, long long (&q)[PER], unsigned &win, int (&eprev)[PER],
    int *fast_e = nullptr)
{
    if (fast_e) *fast_e = -1;
    {
        const double Aend = __dadd_rn(Abefore, own);
        const double c = 2.0 * static_cast<double>(i0 + PER) + 2.0 * static_cast<double>(T) + 160.0;
        const double lo = fmax(__dsub_rn(Abefore, c * ulp_of(Abefore)), Mbefore);
        const double hi = __dadd_rn(Aend, c * ulp_of(Aend));
        const int e = biased_exp(lo);
        if (lo > 0.0 && e != 0x7ff && biased_exp(hi) == e) {
            win = 0;
#pragma unroll
            for (int k = 0; k < PER; ++k) {
                bool ev;
                q[k] = grid_increment(xv[k], e, ev);  // xv is 0 past n: q = 0, no event
                eprev[k] = e;
                if (ev) {
                    q[k] = 0;
                    win |= 1u << k;
                }
            }
            if (fast_e) *fast_e = e;
            return;
        }
    }
    // A zero sum lies on the grid of binade 0 (the subnormals'), so a stretch
    // of leading zeros is a run, not a window per element.
    int ep;
    if (i0 == 0) {
        ep = (s0 >= 0.0 && biased_exp(s0) != 0x7ff) ? biased_exp(s0) : -1;  // s0 itself is exact
    } else {
        ep = certain_binade(Abefore, i0 - 1, T, Mbefore);
    }
    double A = Abefore, M = Mbefore;
    win = 0;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        const uint64_t j = i0 + k;
        q[k] = 0;
        eprev[k] = ep;
        if (j < n) {
            A = __dadd_rn(A, xv[k]);
            M = fmax(M, xv[k]);
            // a zero term leaves the sum unchanged (S_j = S_{j-1}): it keeps
            // the previous binade, certain or not, and is never a window; a
            // run of zeros alone adds nothing, so the walk needs no binade
            // for it
            if (xv[k] == 0.0) continue;
            const int ej = certain_binade(A, j, T, M);
            bool ev = true;
            if (ej >= 0 && ej == ep) q[k] = grid_increment(xv[k], ej, ev);
            if (ev) {
                q[k] = 0;
                win |= 1u << k;
            }
            ep = ej;
        }
    }
}

}  // namespace mckl_b200
