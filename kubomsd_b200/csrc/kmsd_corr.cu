// Spectral velocity-autocorrelation tables without the stored left chain
// (the correlation reduction of src/kubo_msd/solvers/spectral.py:33-38) and
// the per-node Bessel / product-rule tail (spectral.py:39-51) on the device.
//
// tables[b, j, k] = sum_n conj(T_j(Ht) c)[n, b] * cov[n, k, b] for j < length
// and k < kcols, where cov holds the velocity applied to the right chain
// T_k(Ht) v.  The left chain is generated into a ring of kRing vector blocks
// by the engine's fused Chebyshev step; every kRing steps one contraction
// launch reduces the ring against cov:
//   * corr_partial_kernel: CTA (row chunk, tile of k); each thread owns one
//     column b, 8 chain vectors and 4 values of k, and walks the rows of its
//     chunk; partial sums per chunk;
//   * corr_reduce_kernel: tables = sum over chunks in a fixed order.
// Row ownership and the order of the sums are fixed, so the tables are the same
// in every run.  HBM per ring: the ring written once by the steps and read once
// here, and cov read once per k tile.
#include <algorithm>
#include <cstring>
#include <vector>

#include "kmsd.h"
#include "kmsd_impl.h"
#include "kmsd_kernels.cuh"

using namespace kmsd;

namespace {

constexpr int kRing = 32;  // left-chain vector blocks held at once
constexpr int kJT = 8;     // chain vectors of a thread
constexpr int kKT = 4;     // right-chain terms of a thread
constexpr int kJG = kRing / kJT;
constexpr int kCorrThreads = 352;  // most threads of a CTA (184 registers each)
constexpr int kStages = 3;

__device__ __forceinline__ void copy16(void *smem, const void *global) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(global) : "memory");
}

// partial[chunk][jj][k][b] for the ring's chain vectors jj < jn (ring slot
// (j0 + jj) % kRing), rows [chunk * rows_per, ...).
//
// The contraction is FP64-bound: 8 flops per (row, j, k, b), 1.4 GFLOP per ring
// of 16,384 rows, 41 terms and 8 columns, 40 us at the measured 34 TFLOP/s.  A
// CTA takes all 32 chain vectors of its rows, so that cov is read once; a thread
// holds an 8 x 4 tile of sums (128 registers), which needs 12 operand loads for
// 128 multiply-adds; the operands of the next `rs` rows come in with cp.async
// while these are multiplied.  One thread per (k, 8 vectors) without staging, a
// quarter of the vectors per CTA, took 282 us here; this takes 91.
__global__ void __launch_bounds__(kCorrThreads, 1) corr_partial_kernel(const double2 *ring, int64_t slab,
                                                                       const double2 *cov, int64_t n, int nb, int nbp,
                                                                       int k1, int kw, int64_t j0, int jn,
                                                                       int64_t rows_per, int ktiles, int rs,
                                                                       double2 *partial) {
    extern __shared__ __align__(16) double2 stage[];  // kStages x ([kRing][rs][nb], [rs][kw][nb])
    const int chunk = blockIdx.x / ktiles, tile = blockIdx.x % ktiles;
    const int t = threadIdx.x;
    // neighbouring lanes: columns, then terms, then chain vectors
    const int kgroups = (kw + kKT - 1) / kKT;
    const int b = t % nbp, kg = t / nbp % kgroups, jg = t / nbp / kgroups;
    const int kbase = tile * kw, kn = min(kw, k1 - kbase);
    const bool active = b < nb && jg * kJT < jn;
    const int64_t r0 = (int64_t)chunk * rows_per, r1 = min(n, r0 + rows_per);
    const int tsize = kRing * rs * nb, ssize = tsize + rs * kw * nb;
    double2 acc[kJT][kKT];
#pragma unroll
    for (int jj = 0; jj < kJT; ++jj)
#pragma unroll
        for (int i = 0; i < kKT; ++i) acc[jj][i] = make_double2(0., 0.);
    auto fetch = [&](int64_t r, int slot) {  // rows [r, r + rs) into a stage
        if (r < r1) {
            const int rows = (int)min((int64_t)rs, r1 - r), tn = rows * nb, cn = kn * nb;
            double2 *ts = stage + (size_t)slot * ssize, *cs = ts + tsize;
            for (int i = t; i < jn * tn; i += blockDim.x) {
                const int jj = i / tn, x = i - jj * tn;
                copy16(ts + jj * rs * nb + x, ring + (size_t)((j0 + jj) % kRing) * slab + r * nb + x);
            }
            for (int i = t; i < rows * cn; i += blockDim.x) {
                const int row = i / cn, x = i - row * cn;
                copy16(cs + row * kw * nb + x, cov + ((r + row) * k1 + kbase) * nb + x);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int q = 0; q < kStages - 1; ++q) fetch(r0 + (int64_t)q * rs, q);
    int slot = 0;
    for (int64_t r = r0; r < r1; r += rs) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
        __syncthreads();  // this stage is in, and the one before it has been read by all
        fetch(r + (int64_t)(kStages - 1) * rs, (slot + kStages - 1) % kStages);
        if (active) {
            const int rows = (int)min((int64_t)rs, r1 - r);
            const double2 *ts = stage + (size_t)slot * ssize + jg * kJT * rs * nb + b;
            const double2 *cs = stage + (size_t)slot * ssize + tsize + kg * kKT * nb + b;
            for (int row = 0; row < rows; ++row) {
                double2 kv[kKT];
#pragma unroll
                for (int i = 0; i < kKT; ++i) kv[i] = cs[(row * kw + min(i, kn - 1 - kg * kKT)) * nb];
#pragma unroll
                for (int jj = 0; jj < kJT; ++jj) {
                    const double2 cv = ts[(jj * rs + row) * nb];
#pragma unroll
                    for (int i = 0; i < kKT; ++i) {
                        // conj(cv) * kv
                        acc[jj][i].x = fma(cv.x, kv[i].x, fma(cv.y, kv[i].y, acc[jj][i].x));
                        acc[jj][i].y = fma(cv.x, kv[i].y, fma(-cv.y, kv[i].x, acc[jj][i].y));
                    }
                }
            }
        }
        slot = slot + 1 == kStages ? 0 : slot + 1;
    }
    if (!active) return;
    double2 *out = partial + (size_t)chunk * kRing * k1 * nb;
#pragma unroll
    for (int jj = 0; jj < kJT; ++jj) {
        if (jg * kJT + jj >= jn) break;
#pragma unroll
        for (int i = 0; i < kKT; ++i) {
            const int k = kg * kKT + i;
            if (k < kn) out[((size_t)(jg * kJT + jj) * k1 + kbase + k) * nb + b] = acc[jj][i];
        }
    }
}

// tables[b][j0 + jj][k] = sum over chunks of partial: a CTA takes 32 elements,
// eight threads each, which sum every eighth chunk; their sums are joined in
// order.
__global__ void __launch_bounds__(256) corr_reduce_kernel(const double2 *partial, int nchunks, int jn, int k1, int nb,
                                                          int64_t j0, int64_t length, double2 *tables) {
    __shared__ double2 part[8][32];
    const int64_t total = (int64_t)jn * k1 * nb;
    const size_t stride = (size_t)kRing * k1 * nb;
    const int x = threadIdx.x & 31, q = threadIdx.x >> 5;
    for (int64_t e0 = blockIdx.x * (int64_t)32; e0 < total; e0 += (int64_t)gridDim.x * 32) {
        const int64_t e = e0 + x;
        double2 s = make_double2(0., 0.);
        if (e < total) {
#pragma unroll 4
            for (int c = q; c < nchunks; c += 8) {
                const double2 v = partial[c * stride + e];
                s.x += v.x;
                s.y += v.y;
            }
        }
        part[q][x] = s;
        __syncthreads();
        if (q == 0 && e < total) {
#pragma unroll
            for (int i = 1; i < 8; ++i) {
                s.x += part[i][x].x;
                s.y += part[i][x].y;
            }
            const int b = (int)(e % nb);
            const int64_t jk = e / nb;
            const int k = (int)(jk % k1), jj = (int)(jk / k1);
            tables[((size_t)b * length + j0 + jj) * k1 + k] = s;
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------ node tail
// For the spectral nodes t_m of one segment, with Bessel coefficients
// coef[m][p] (p <= kt[m]):
//   q[m][b][j]   = sum_{k <= kt[m]} tables[b][j][k] coef[m][k]          (j < L + kt[m])
//   mom[m][b][l] = Re sum_{p <= kt[m]} (q[l + p] + q[|l - p|]) / 2 conj(coef[m][p])   (l < L)
//   vac[m][b][e] = sum_l G[e][l] mom[m][b][l]
// (the product rule T_l T_p = (T_{l+p} + T_|l-p|) / 2 of spectral.py:43-49).
__global__ void node_q_kernel(const double2 *tables, int nb, int64_t length, int k1, const double2 *coef,
                              const int *kt, int m, int64_t L, double2 *q) {
    const int64_t total = (int64_t)m * nb * length;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t j = e % length;
        const int64_t mb = e / length;
        const int b = (int)(mb % nb), node = (int)(mb / nb);
        const int K = kt[node];
        double sx = 0., sy = 0.;
        if (j < L + K) {
            const double2 *tr = tables + ((size_t)b * length + j) * k1;
            const double2 *cr = coef + (size_t)node * k1;
            for (int k = 0; k <= K; ++k) {
                const double2 tv = tr[k], cv = cr[k];
                sx = fma(tv.x, cv.x, fma(-tv.y, cv.y, sx));
                sy = fma(tv.x, cv.y, fma(tv.y, cv.x, sy));
            }
        }
        q[e] = make_double2(sx, sy);
    }
}

__global__ void node_moments_kernel(const double2 *q, int nb, int64_t length, int k1, const double2 *coef,
                                    const int *kt, int m, int64_t L, double *mom) {
    const int64_t total = (int64_t)m * nb * L;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t l = e % L;
        const int64_t mb = e / L;
        const int node = (int)(mb / nb);
        const int K = kt[node];
        const double2 *qr = q + mb * length;
        const double2 *cr = coef + (size_t)node * k1;
        double s = 0.;
        for (int p = 0; p <= K; ++p) {
            const double2 a = qr[l + p], c = qr[l >= p ? l - p : p - l], cv = cr[p];
            // Re((a + c) / 2 * conj(cv))
            s += .5 * ((a.x + c.x) * cv.x + (a.y + c.y) * cv.y);
        }
        mom[e] = s;
    }
}

// vac[row][e] = sum_l G[e][l] mom[row][l]; one warp per (row, e).
__global__ void node_project_kernel(const double *mom, int64_t rows, int64_t L, const double *G, int ne,
                                    double *vac) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x / 32);
    for (int64_t w = blockIdx.x * (int64_t)(blockDim.x / 32) + threadIdx.x / 32; w < rows * ne; w += warps) {
        const int64_t row = w / ne;
        const int e = (int)(w % ne);
        const double *mr = mom + row * L, *gr = G + (size_t)e * L;
        double s = 0.;
        for (int64_t l = lane; l < L; l += 32) s = fma(gr[l], mr[l], s);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) vac[w] = s;
    }
}

}  // namespace

namespace kmsd {

// One contraction of the ring's chain vectors [j0, j0 + jn) against cov.
int corr_ring(const double2 *ring, int64_t n, int nb, const double2 *cov, int k1, int64_t j0, int jn,
              int64_t length, double2 *tables, DevBuf &partial, cudaStream_t s) {
    const int nbp = nb <= 1 ? 1 : nb <= 2 ? 2 : nb <= 4 ? 4 : 8;
    if (nb > 8 || k1 > 4 * (256 / nbp))
        return fail(KMSD_EINVAL, "correlation tables take at most 8 vectors and 1024/vectors right-chain terms per call");
    // terms of a CTA: what its threads hold, shared evenly among the k tiles
    const int most = kCorrThreads / (nbp * kJG) * kKT, ktiles = (k1 + most - 1) / most;
    const int kw = (((k1 + ktiles - 1) / ktiles) + kKT - 1) / kKT * kKT;
    const int threads = (nbp * kJG * (kw / kKT) + 31) / 32 * 32;
    // rows of a stage: three stages in about 200 KB, at most 16 rows each
    const size_t row_bytes = (size_t)(kRing + kw) * nb * sizeof(double2);
    const int rs = (int)std::max<size_t>(1, std::min<size_t>(16, 200 * 1024 / kStages / row_bytes));
    const size_t smem = kStages * rs * row_bytes;
    int nchunks = (int)std::max<int64_t>(1, std::min<int64_t>(std::max(1, sm_count() / ktiles), (n + rs - 1) / rs));
    const int64_t rows_per = (n + nchunks - 1) / nchunks;
    nchunks = (int)((n + rows_per - 1) / rows_per);
    if (partial.ensure((size_t)nchunks * kRing * k1 * nb * sizeof(double2))) return KMSD_ECUDA;
    static PerDevice<cudaError_t> attr;
    KMSD_CUDA(attr.get([](int) {
        return cudaFuncSetAttribute((const void *)corr_partial_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    200 * 1024);
    }));
    corr_partial_kernel<<<nchunks * ktiles, threads, smem, s>>>(ring, n * nb, cov, n, nb, nbp, k1, kw, j0, jn, rows_per,
                                                                ktiles, rs, partial.as<double2>());
    count_launch();
    const int64_t total = (int64_t)jn * k1 * nb;
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((total + 31) / 32, (int64_t)sm_count() * 16));
    corr_reduce_kernel<<<grid, 256, 0, s>>>(partial.as<double2>(), nchunks, jn, k1, nb, j0, length, tables);
    count_launch();
    KMSD_CUDA(cudaGetLastError());
    return KMSD_OK;
}

int ring_slots() { return kRing; }

}  // namespace kmsd

extern "C" int kmsd_vac_nodes(const void *tables, int64_t b, int64_t length, int64_t kcols, int64_t n_moments,
                              const void *coeff, const int *orders, int64_t nodes, const double *G,
                              int64_t n_energy, void *work, int64_t work_bytes, double *vac, void *stream) {
    if (!tables || !coeff || !orders || !G || !vac || b < 1 || nodes < 1 || n_energy < 1 || n_moments < 1 ||
        kcols < 1 || length < n_moments)
        return fail(KMSD_EINVAL, "invalid spectral node arguments");
    const int64_t need = nodes * b * length * (int64_t)sizeof(double2) + nodes * b * n_moments * 8;
    if (!work || work_bytes < need) return fail(KMSD_EINVAL, "spectral node workspace too small");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    double2 *q = static_cast<double2 *>(work);
    double *mom = reinterpret_cast<double *>(q + nodes * b * length);
    auto grid_of = [](int64_t total) {
        return (int)std::max<int64_t>(1, std::min<int64_t>((total + 255) / 256, (int64_t)sm_count() * 8));
    };
    node_q_kernel<<<grid_of(nodes * b * length), 256, 0, s>>>(static_cast<const double2 *>(tables), (int)b, length,
                                                              (int)kcols, static_cast<const double2 *>(coeff), orders,
                                                              (int)nodes, n_moments, q);
    count_launch();
    node_moments_kernel<<<grid_of(nodes * b * n_moments), 256, 0, s>>>(q, (int)b, length, (int)kcols,
                                                                       static_cast<const double2 *>(coeff), orders,
                                                                       (int)nodes, n_moments, mom);
    count_launch();
    const int64_t warps = nodes * b * n_energy;
    node_project_kernel<<<(int)std::max<int64_t>(1, std::min<int64_t>((warps + 7) / 8, (int64_t)sm_count() * 8)),
                          256, 0, s>>>(mom, nodes * b, n_moments, G, (int)n_energy, vac);
    count_launch();
    KMSD_CUDA(cudaGetLastError());
    return KMSD_OK;
}
