// Chebyshev moments of a small operator in one launch (kmsd_cluster.cu).
#pragma once

#include "kmsd_impl.h"
#include "kmsd_kernels.cuh"

namespace kmsd {

// One independent system: rows [row0, row0 + n) of the operator and of the
// vector block, its spectral window and its moments (length x b, row-major).
struct ClusterSystem {
    int64_t row0;
    int64_t n;
    double center, half;
    double *mu;
};

// Rows of at most this many real entries are kept in registers.
constexpr int kClusterWidth = 8;

// How the moments of systems of up to n rows and b columns are computed by this
// path; size 0 where it does not apply.
struct ClusterPlan {
    int size = 0;   // CTAs per cluster
    int rows = 0;   // rows of a CTA
    int cols = 0;   // columns of a cluster
    int groups = 0; // clusters per system
    int rpt = 0, threads = 0, cg = 0;
    size_t smem = 0;
};
template <class T>
int cluster_plan(int64_t n, int width, int64_t b, bool doubling, int64_t systems, ClusterPlan *out);
// Bytes of device scratch a planned call needs.
size_t cluster_scratch(const ClusterPlan &pl, int64_t systems, int64_t length, bool doubling);
// Queues the moments of `systems` (a device array; one: `one` by value instead).
template <class T>
int cluster_moments(const ClusterPlan &pl, const CsrView<T> &H, int width, const double2 *B, int64_t b, int64_t length,
                    bool doubling, const ClusterSystem *systems, int64_t count, const ClusterSystem &one, double *scratch,
                    cudaStream_t s);

}  // namespace kmsd
