// Chebyshev moments of a small operator in one launch (kmsd_cluster.cu).
#pragma once

#include <vector>

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

// The columns [c0, c0 + cols) of a system: the work of one cluster.
struct ClusterJob {
    int system, c0, cols, pad;
};

// Rows of at most this many real entries are kept in registers.
constexpr int kClusterWidth = 8;

// How moments are computed by this path; size 0 where it does not apply.
struct ClusterPlan {
    int size = 0;    // CTAs per cluster
    int cols = 0;    // (most) columns of a cluster
    int groups = 0;  // clusters
    int rpt = 0, threads = 0, cg = 0;
    size_t smem = 0;
};
// One system of n rows of up to `width` entries; several (rows_of), with the
// work of each cluster.
template <class T> int cluster_plan(int64_t n, int width, int64_t b, bool doubling, ClusterPlan *out);
template <class T>
int cluster_batch_plan(const std::vector<int64_t> &rows_of, int width, int64_t b, bool doubling, ClusterPlan *out,
                       std::vector<ClusterJob> *jobs);
// Bytes of device scratch a planned call needs.
size_t cluster_scratch(const ClusterPlan &pl, int64_t length, bool doubling);
// Queues the moments (length >= 2) of `one`, or of `systems` by `jobs` (device arrays).
template <class T>
int cluster_moments(const ClusterPlan &pl, const CsrView<T> &H, int width, const double2 *B, int64_t b, int64_t length,
                    bool doubling, const ClusterSystem *systems, const ClusterJob *jobs, const ClusterSystem &one,
                    double *scratch, cudaStream_t s);

}  // namespace kmsd
