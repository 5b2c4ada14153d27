// Recurrences of small operators in one launch of thread-block clusters: moments
// (kmsd_cluster.cu) and the Bessel series (kmsd_cluster_series.cu).
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

// ---------------------------------------------------------------- shared parts
template <class T> struct Cx;
template <> struct Cx<double> { using type = double2; };
template <> struct Cx<float> { using type = float2; };

// Threads that own rows (one more warp sums): what 96 (complex64) or 128
// (complex128) registers a thread allow.
template <class T> constexpr int kMaxCompute = sizeof(T) == 4 ? 608 : 480;

// The cluster's meeting in two halves: what lies between them overlaps the
// meeting and becomes visible with the next one.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ void cluster_sync_all() {
    cluster_arrive();
    cluster_wait();
}
__device__ __forceinline__ unsigned remote_address(unsigned at, unsigned rank) {
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(at), "r"(rank));
    return r;
}
// An element from any CTA's shared memory, this one's too: addresses of the own
// CTA take the same load at the same speed, so no read needs a branch (one branch
// per row made 4,096 x 8 4 % and 16,129 x 31 7 % slower).
__device__ __forceinline__ double2 load_any(unsigned at, double2) {
    double2 v;
    asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(at));
    return v;
}
__device__ __forceinline__ float2 load_any(unsigned at, float2) {
    float2 v;
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(at));
    return v;
}

// Sets of warps that share out a cluster's columns (1: all warps own rows).
__host__ __device__ inline int column_sets(int warps, int rows) {
    const int wr = rows > 32 ? (rows + 31) / 32 : 1;
    return 2 * wr <= warps ? warps / wr : 1;
}

// Dynamic shared memory a CTA may have on this device.
size_t cluster_smem_limit();
// Launch configuration of `ctas` CTAs in clusters of `size`; `at` has one entry.
void cluster_config(cudaLaunchConfig_t &cfg, cudaLaunchAttribute *at, int ctas, int size, int threads, size_t smem);
// Clusters of this shape that run at once (cached; also sets the kernel's
// attributes on first use).
int active_clusters(const void *kernel, int size, int threads, size_t smem);

// ---------------------------------------------------------------- series
// Most coefficients of a series taken by this path (they travel in the launch).
constexpr int kSeriesTerms = 192;
// How a series of columns psi (with their phi block: `phi`) is computed.
template <class T> int series_plan(int64_t n, int width, int64_t nb, bool phi, ClusterPlan *out);
// Queues out = sum_k coeff[k] T_k(A) B over the columns [0, nb) (psi) and, with
// vim (the imaginary entries of a purely imaginary velocity in H's CSR order) the
// columns [phi0, phi0 + nb) (phi) of the (n, b) arrays; wi is the weight of the
// injection wi i V psi.  psi columns are written when write_psi is set.
template <class T>
int cluster_series(const ClusterPlan &pl, const CsrView<T> &H, int width, int64_t n, const T *vim, double wi,
                   const double2 *B, double2 *out, int64_t b, int64_t nb, int64_t phi0, bool write_psi,
                   const double *coeff, int64_t ncoeff, double center, double half, int *status, cudaStream_t s);

// How a stored chain of b columns is computed.
template <class T> int chain_plan(int64_t n, int width, int64_t b, ClusterPlan *out);
// Queues T_k for k0 <= k < k1 from cur = T_{k0-1} and prev = T_{k0-2} (nullptr:
// k0 is 1), all (n, b) complex128, into store + (ring ? k % ring : k) * n * b; cur
// and prev may be blocks of that ring.
template <class T>
int cluster_chain(const ClusterPlan &pl, const CsrView<T> &H, int width, int64_t n, const double2 *cur, const double2 *prev,
                  double2 *store, int ring, int64_t b, int64_t k0, int64_t k1, double center, double half, cudaStream_t s);

}  // namespace kmsd
