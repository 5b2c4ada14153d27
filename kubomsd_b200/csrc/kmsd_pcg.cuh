// Per-column state of the batched PCG, shared by its two drivers: the launch
// sequence of kmsd_metric.cu and the resident solve of kmsd_pcg.cu.
#pragma once

#include "kmsd.h"
#include "kmsd_impl.h"
#include "kmsd_kernels.cuh"

namespace kmsd {

struct ColPtr {
    double *safe, *bn, *thr, *rz, *alpha, *beta, *rn, *tn, *newrz, *gap, *relative, *residual;
    double *rsn;  // residual norm at the last (re)start (mixed form)
    int *active, *restart, *brk, *conv, *finp, *fino;
    long long *iters;
    int *flags;  // [0] halt, [1] check, [2] nonfinite rhs, [3] breakdown, [4] n_active
};
constexpr int kDoubles = 13, kInts = 6;
inline size_t col_bytes(int64_t b) { return (size_t)b * (kDoubles * 8 + kInts * 4 + 8) + 64; }
inline ColPtr col_ptr(void *base, int64_t b) {
    ColPtr c;
    double *d = static_cast<double *>(base);
    double **dp[kDoubles] = {&c.safe, &c.bn, &c.thr, &c.rz, &c.alpha, &c.beta,       &c.rn,
                             &c.tn,   &c.newrz, &c.gap, &c.relative, &c.residual, &c.rsn};
    for (int i = 0; i < kDoubles; ++i) *dp[i] = d + (size_t)i * b;
    long long *l = reinterpret_cast<long long *>(d + (size_t)kDoubles * b);
    c.iters = l;
    int *ip = reinterpret_cast<int *>(l + b);
    int **ipp[kInts] = {&c.active, &c.restart, &c.brk, &c.conv, &c.finp, &c.fino};
    for (int i = 0; i < kInts; ++i) *ipp[i] = ip + (size_t)i * b;
    c.flags = ip + (size_t)kInts * b;
    return c;
}
// device counters: [0] refreshes [1] checks [2] restarts [3] iterations sum; max
// relative residual; continuations of one-launch solves
struct Counters {
    long long v[4];
    double max_rel;
    long long redos;
};

struct Pre {
    const double *diag;
    const int *bstart;
    const int64_t *foff;
    const double2 *factors;
    int ub;    // uniform block size, or 0: rows and factors are then found without lookups
    int real;  // every block inverse is real
};

// One whole solve as a single launch (kmsd_pcg.cu).  `resident_plan` decides
// whether it applies to b columns of M (and to which of its forms), sizes and
// allocates its scratch; `resident_solve` queues it on s and allocates nothing.
struct ResidentPlan {
    int form = 0;  // 0: does not apply
    int ctas = 0, threads = 0;
    size_t smem = 0;
    int lcw = 0, lks = 0, nch = 1;  // log2 of a chunk's columns and of the lanes that split a block row; chunks
    int own = 0, blocks = 0;                     // block rows and S blocks of the largest CTA share
    const kmsd_metric_s::Halo *halo = nullptr;  // of the forms that stage it
};
int resident_plan(kmsd_metric_s *M, int64_t b, ResidentPlan *out);
int resident_solve(kmsd_metric_s *M, const ResidentPlan &pl, const double2 *B, double2 *Y, int64_t b, double rtol,
                   double atol, int maxiter, cudaStream_t s, int *status, FailReportFull *fr);

}  // namespace kmsd
