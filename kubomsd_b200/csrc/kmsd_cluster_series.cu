// The Bessel series and stored Chebyshev chains of small orthogonal-basis
// operators in one launch.
//
// Series: the propagation sum_k c_k T_k(A) of psi columns, alone or with the phi
// block of one direction whose velocity is purely imaginary (the lattice velocities
// i H_ij dx_ij / hbar).
//
// As kmsd_cluster.cu: a thread-block cluster takes a few psi columns and their phi
// columns through all terms, with T_k, T_{k-1} and the accumulator in shared
// memory and the entries of H and V in registers; psi's neighbours serve H psi
// and V psi.  The launch sequence takes 24 to 90 launches of 4 to 11 us here.
// 43 terms of [psi | phi], 2 x 8 complex128 columns: 64 x 64 sites 0.08 ms
// against 0.36 ms.  The arithmetic of an element is that of cheb_step_kernel's
// series epilogue.
#include <algorithm>
#include <cstring>
#include <map>
#include <mutex>
#include <tuple>

#include "kmsd_cluster.cuh"

using namespace kmsd;

namespace {

template <class T> struct SeriesArgs {
    CsrView<T> H;
    const T *vim;
    const double2 *B;
    double2 *out;
    int64_t n, b, nb, phi0;
    int write_psi;
    int cols, terms;
    double center, half;
    T wi;
    int *status;
    T coeff[2 * kSeriesTerms];
};

// Products and sums rounded by themselves: t, the injection and their sum are
// three roundings, as in the step kernel.
__device__ __forceinline__ double times(double x, double y) { return __dmul_rn(x, y); }
__device__ __forceinline__ float times(float x, float y) { return __fmul_rn(x, y); }
__device__ __forceinline__ double plus(double x, double y) { return __dadd_rn(x, y); }
__device__ __forceinline__ float plus(float x, float y) { return __fadd_rn(x, y); }

// Rows of up to W entries, RPT rows per thread; PHI: with a phi block.
template <class T, int W, int RPT, bool PHI>
__global__ void __launch_bounds__(kMaxCompute<T>, 1) cluster_series_kernel(const __grid_constant__ SeriesArgs<T> a) {
    using V = typename Cx<T>::type;
    constexpr int BLK = PHI ? 2 : 1;
    extern __shared__ __align__(16) unsigned char sm[];
    unsigned rank, size;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(size));
    const int c0 = (int)(blockIdx.x / size) * a.cols, cols = min(a.cols, (int)(a.nb - c0));
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, compute = blockDim.x;
    const int rows = (int)((a.n + size - 1) / size);
    const int mine = max(0, min(rows, (int)(a.n - (int64_t)rank * rows)));
    const int cwarps = compute / 32, wr = max(1, (rows + 31) / 32), sets = column_sets(cwarps, rows);
    const int set = sets > 1 ? warp / wr : 0, own = sets > 1 ? warp - set * wr : warp;
    const int at_row = own * 32 + lane;
    const bool works = set < sets && own < min(cwarps, (mine + 31) / 32) && set < cols;
    // [T_{k-1} | T_k | sum][psi, phi][column][row]
    const unsigned plane = (unsigned)rows * sizeof(V), half_block = plane * cols, block = half_block * BLK;
    const unsigned base = (unsigned)__cvta_generic_to_shared(sm);
    V *vec = reinterpret_cast<V *>(sm);
    const int64_t g0 = (int64_t)rank * rows;

    unsigned at[RPT][W];
    T val[RPT][W], vel[RPT][PHI ? W : 1];
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
        const int r = i * compute + at_row;
        const bool on = works && r < mine;
        const int k0 = on ? a.H.ptr[g0 + r] : 0, k1 = on ? a.H.ptr[g0 + r + 1] : 0;
#pragma unroll
        for (int j = 0; j < W; ++j) {
            at[i][j] = base + (on ? (unsigned)r * (unsigned)sizeof(V) : 0u);
            val[i][j] = T(0);
            if (PHI) vel[i][PHI ? j : 0] = T(0);
            if (k0 + j < k1) {
                const int c = a.H.idx[k0 + j], owner = c / rows, loc = c - owner * rows;
                val[i][j] = a.H.re[k0 + j];
                if (PHI) vel[i][PHI ? j : 0] = a.vim[k0 + j];
                at[i][j] = base + (unsigned)loc * (unsigned)sizeof(V);
                if (owner != (int)rank) at[i][j] = remote_address(at[i][j], owner);
            }
        }
    }
    for (int i = tid; i < mine * cols; i += blockDim.x) {
        const int r = i / cols, c = i - r * cols;
#pragma unroll
        for (int q = 0; q < BLK; ++q) {
            const double2 v = a.B[(g0 + r) * a.b + (q ? a.phi0 : 0) + c0 + c];
            V w;
            w.x = (T)v.x;
            w.y = (T)v.y;
            vec[(size_t)(q * cols + c) * rows + r] = w;
            w.x = w.y = T(0);
            vec[(size_t)((BLK + q) * cols + c) * rows + r] = w;  // "T_{-1}": the first step is t - 0
        }
    }
    cluster_sync_all();

    const T cen = (T)a.center, hal = (T)a.half, inv = (T)(1. / a.half);
    unsigned cur = 0;  // offset of T_{k-1}; T_k goes to the other block, over T_{k-2}
    T two = T(1);      // 2, and 1 in the first step
    for (int k = 1; k < a.terms; ++k) {
        if (works) {
            const unsigned nxt = block - cur;
            const T ckr = a.coeff[2 * k], cki = a.coeff[2 * k + 1];
            for (int c = set; c < cols; c += sets) {
#pragma unroll
                for (int i = 0; i < RPT; ++i) {
                    const int r = i * compute + at_row;
                    if (r < mine) {
                        V inject;
                        inject.x = inject.y = T(0);
#pragma unroll
                        for (int q = 0; q < BLK; ++q) {
                            const unsigned off = (unsigned)q * half_block + (unsigned)c * plane;
                            const unsigned me = off + (unsigned)r * (unsigned)sizeof(V);
                            V xv[W];
#pragma unroll
                            for (int j = 0; j < W; ++j) xv[j] = load_any(at[i][j] + off + cur, V{});
                            const V x = *reinterpret_cast<const V *>(sm + me + cur);
                            V *dst = reinterpret_cast<V *>(sm + me + nxt), *sum = reinterpret_cast<V *>(sm + me + 2 * block);
                            const V pv = *dst, ov = *sum;
                            V h;
                            h.x = h.y = T(0);
#pragma unroll
                            for (int j = 0; j < W; ++j) {
                                h.x = fma(val[i][j], xv[j].x, h.x);
                                h.y = fma(val[i][j], xv[j].y, h.y);
                            }
                            T tr = rdiv(h.x - cen * x.x, hal, inv), ti = rdiv(h.y - cen * x.y, hal, inv);
                            if (PHI) {
                                if (q == 0) {
                                    V vp;  // V psi for purely imaginary V
                                    vp.x = vp.y = T(0);
#pragma unroll
                                    for (int j = 0; j < W; ++j) {
                                        vp.x = fma(-vel[i][PHI ? j : 0], xv[j].y, vp.x);
                                        vp.y = fma(vel[i][PHI ? j : 0], xv[j].x, vp.y);
                                    }
                                    inject.x = -times(a.wi, vp.y);
                                    inject.y = times(a.wi, vp.x);
                                } else {
                                    tr = plus(tr, inject.x);
                                    ti = plus(ti, inject.y);
                                }
                            }
                            V nx;
                            nx.x = fma(two, tr, -pv.x);
                            nx.y = fma(two, ti, -pv.y);
                            *dst = nx;
                            V o;
                            if (k == 1) {
                                o.x = a.coeff[0] * x.x - a.coeff[1] * x.y + ckr * nx.x - cki * nx.y;
                                o.y = a.coeff[0] * x.y + a.coeff[1] * x.x + ckr * nx.y + cki * nx.x;
                            } else {
                                o = ov;
                                o.x += ckr * nx.x - cki * nx.y;
                                o.y += ckr * nx.y + cki * nx.x;
                            }
                            *sum = o;
                        }
                    }
                }
            }
        }
        cluster_sync_all();
        cur = block - cur;
        two = T(2);
    }
    // a nonfinite value of any term stays in the sum
    bool bad = false;
    for (int i = tid; i < mine * cols; i += blockDim.x) {
        const int r = i / cols, c = i - r * cols;
#pragma unroll
        for (int q = 0; q < BLK; ++q) {
            const V v = vec[(size_t)((2 * BLK + q) * cols + c) * rows + r];
            bad |= !isfinite(v.x) || !isfinite(v.y);
            if (q || a.write_psi)
                a.out[(g0 + r) * a.b + (q ? a.phi0 : 0) + c0 + c] = make_double2((double)v.x, (double)v.y);
        }
    }
    if (bad) atomicOr(a.status, 1);
}

template <class T> struct ChainArgs {
    CsrView<T> H;
    const double2 *cur, *prev;  // T_{k0-1}, T_{k0-2} (nullptr: k0 is 1)
    double2 *store;             // T_k goes to store + (ring ? k % ring : k) * n * b
    int64_t n, b;
    int ring, cols;
    int64_t k0, k1;
    double center, half;
};

// T_k for k0 <= k < k1, every one stored.  The stores are issued between the two
// halves of the meeting, so that the next arrival finds them under way for a
// step (a meeting right behind global stores takes four times as long).
template <class T, int W, int RPT>
__global__ void __launch_bounds__(kMaxCompute<T>, 1) cluster_chain_kernel(const ChainArgs<T> a) {
    using V = typename Cx<T>::type;
    extern __shared__ __align__(16) unsigned char sm[];
    unsigned rank, size;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(size));
    const int c0 = (int)(blockIdx.x / size) * a.cols, cols = min(a.cols, (int)(a.b - c0));
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, compute = blockDim.x;
    const int rows = (int)((a.n + size - 1) / size);
    const int mine = max(0, min(rows, (int)(a.n - (int64_t)rank * rows)));
    const int cwarps = compute / 32, wr = max(1, (rows + 31) / 32), sets = column_sets(cwarps, rows);
    const int set = sets > 1 ? warp / wr : 0, own = sets > 1 ? warp - set * wr : warp;
    const int at_row = own * 32 + lane;
    const bool works = set < sets && own < min(cwarps, (mine + 31) / 32) && set < cols;
    // [T_{k-1} | T_k][column][row]
    const unsigned plane = (unsigned)rows * sizeof(V), block = plane * cols;
    const unsigned base = (unsigned)__cvta_generic_to_shared(sm);
    V *vec = reinterpret_cast<V *>(sm);
    const int64_t g0 = (int64_t)rank * rows;

    unsigned at[RPT][W];
    T val[RPT][W];
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
        const int r = i * compute + at_row;
        const bool on = works && r < mine;
        const int k0 = on ? a.H.ptr[g0 + r] : 0, k1 = on ? a.H.ptr[g0 + r + 1] : 0;
#pragma unroll
        for (int j = 0; j < W; ++j) {
            at[i][j] = base + (on ? (unsigned)r * (unsigned)sizeof(V) : 0u);
            val[i][j] = T(0);
            if (k0 + j < k1) {
                const int c = a.H.idx[k0 + j], owner = c / rows, loc = c - owner * rows;
                val[i][j] = a.H.re[k0 + j];
                at[i][j] = base + (unsigned)loc * (unsigned)sizeof(V);
                if (owner != (int)rank) at[i][j] = remote_address(at[i][j], owner);
            }
        }
    }
    for (int i = tid; i < mine * cols; i += blockDim.x) {
        const int r = i / cols, c = i - r * cols;
        const int64_t g = (g0 + r) * a.b + c0 + c;
        const double2 x = a.cur[g], p = a.prev ? a.prev[g] : make_double2(0., 0.);
        V w;
        w.x = (T)x.x;
        w.y = (T)x.y;
        vec[(size_t)c * rows + r] = w;
        w.x = (T)p.x;
        w.y = (T)p.y;
        vec[(size_t)(cols + c) * rows + r] = w;
    }
    cluster_sync_all();

    const T cen = (T)a.center, hal = (T)a.half, inv = (T)(1. / a.half);
    unsigned cur = 0;
    T two = a.prev ? T(2) : T(1);
    for (int64_t k = a.k0; k < a.k1; ++k) {
        const unsigned nxt = block - cur;
        if (works) {
            for (int c = set; c < cols; c += sets) {
#pragma unroll
                for (int i = 0; i < RPT; ++i) {
                    const int r = i * compute + at_row;
                    if (r < mine) {
                        const unsigned off = (unsigned)c * plane, me = off + (unsigned)r * (unsigned)sizeof(V);
                        V xv[W];
#pragma unroll
                        for (int j = 0; j < W; ++j) xv[j] = load_any(at[i][j] + off + cur, V{});
                        const V x = *reinterpret_cast<const V *>(sm + me + cur);
                        V *dst = reinterpret_cast<V *>(sm + me + nxt);
                        const V pv = *dst;
                        V h;
                        h.x = h.y = T(0);
#pragma unroll
                        for (int j = 0; j < W; ++j) {
                            h.x = fma(val[i][j], xv[j].x, h.x);
                            h.y = fma(val[i][j], xv[j].y, h.y);
                        }
                        const T tr = rdiv(h.x - cen * x.x, hal, inv), ti = rdiv(h.y - cen * x.y, hal, inv);
                        V nx;
                        nx.x = fma(two, tr, -pv.x);
                        nx.y = fma(two, ti, -pv.y);
                        *dst = nx;
                    }
                }
            }
        }
        cluster_arrive();
        if (works) {
            double2 *out = a.store + (size_t)(a.ring ? k % a.ring : k) * a.n * a.b;
            for (int c = set; c < cols; c += sets)
#pragma unroll
                for (int i = 0; i < RPT; ++i) {
                    const int r = i * compute + at_row;
                    if (r < mine) {
                        const V v = *reinterpret_cast<const V *>(sm + (unsigned)c * plane + (unsigned)r * (unsigned)sizeof(V) + nxt);
                        out[(g0 + r) * a.b + c0 + c] = make_double2((double)v.x, (double)v.y);
                    }
                }
        }
        cluster_wait();
        cur = nxt;
        two = T(2);
    }
}

template <class T, int W>
const void *pick_chain_rows(int rpt) {
    switch (rpt) {
        case 1: return (const void *)cluster_chain_kernel<T, W, 1>;
        case 2: return (const void *)cluster_chain_kernel<T, W, 2>;
        case 3:
            if constexpr (W < kClusterWidth) return (const void *)cluster_chain_kernel<T, W, 3>;
    }
    return nullptr;
}
template <class T>
const void *pick_chain(int width, int rpt) {
    if (width <= 4) return pick_chain_rows<T, 4>(rpt);
    if (width <= 5) return pick_chain_rows<T, 5>(rpt);
    return pick_chain_rows<T, 8>(rpt);
}

template <class T, int W, bool PHI>
const void *pick_rows(int rpt) {
    switch (rpt) {
        case 1: return (const void *)cluster_series_kernel<T, W, 1, PHI>;
        case 2: return (const void *)cluster_series_kernel<T, W, 2, PHI>;
        case 3:
            if constexpr (W < kClusterWidth && sizeof(T) == 4) return (const void *)cluster_series_kernel<T, W, 3, PHI>;
    }
    return nullptr;
}
template <class T, bool PHI>
const void *pick_width(int width, int rpt) {
    if (width <= 4) return pick_rows<T, 4, PHI>(rpt);
    if (width <= 5) return pick_rows<T, 5, PHI>(rpt);
    return pick_rows<T, 8, PHI>(rpt);
}
template <class T>
const void *pick_kernel(int width, int rpt, bool phi) {
    return phi ? pick_width<T, true>(width, rpt) : pick_width<T, false>(width, rpt);
}

enum { kChain = 0, kPsi = 1, kPsiPhi = 2 };

// The cheapest shape for nb (psi) columns of `what`, as the moments' plan with
// the accumulator and the phi block (cached).
template <class T> int find_plan(int what, int64_t n, int width, int64_t nb, ClusterPlan *out) {
    *out = ClusterPlan{};
    if (width < 1 || width > kClusterWidth) return KMSD_OK;
    static std::mutex lock;
    static std::map<std::tuple<int, int, int64_t, int, int64_t>, ClusterPlan> cache;
    const auto key = std::make_tuple(current_device(), what, n, width, nb);
    const int planes = what == kChain ? 2 : what == kPsi ? 3 : 6, blocks = what == kPsiPhi ? 2 : 1;
    {
        std::lock_guard<std::mutex> guard(lock);
        const auto it = cache.find(key);
        if (it != cache.end()) {
            *out = it->second;
            return KMSD_OK;
        }
    }
    double best = 0.;
    for (int size : {16, 8, 4, 2, 1}) {
        const int64_t rows = (n + size - 1) / size;
        const int rpt = (int)((rows + kMaxCompute<T> - 1) / kMaxCompute<T>);
        const void *kernel = what == kChain ? pick_chain<T>(width, rpt) : pick_kernel<T>(width, rpt, what == kPsiPhi);
        if (!kernel) continue;
        const int threads = (int)(((rows + rpt - 1) / rpt + 31) / 32 * 32), warps = threads / 32;
        const int sets = column_sets(warps, (int)rows);
        for (int cols = 1; cols <= std::min<int64_t>(nb, 32); ++cols) {
            const size_t smem = (size_t)rows * cols * 2 * sizeof(T) * planes;
            if (smem > cluster_smem_limit()) break;
            const int64_t groups = (nb + cols - 1) / cols;
            const int act = active_clusters(kernel, size, threads, smem);
            if (act < 1) continue;
            const int64_t items = (int64_t)((cols + sets - 1) / sets) * rpt * blocks;
            const double traffic = std::min<int64_t>(warps, sets * ((rows + 31) / 32)) * (width + 5.) * (2 * sizeof(T)) * 32 / 128.;
            const double cost = ((size > 1 ? 1000. : 600.) + items * std::max(400., traffic)) * ((groups + act - 1) / act);
            if (out->size == 0 || cost < best) {
                best = cost;
                *out = ClusterPlan{size, cols, (int)groups, rpt, threads, 1, smem};
            }
        }
    }
    std::lock_guard<std::mutex> guard(lock);
    if (cache.size() >= 1024) cache.clear();
    cache[key] = *out;
    return KMSD_OK;
}

}  // namespace

namespace kmsd {

template <class T> int series_plan(int64_t n, int width, int64_t nb, bool phi, ClusterPlan *out) {
    return find_plan<T>(phi ? kPsiPhi : kPsi, n, width, nb, out);
}
// A chain stores n x b complex128 values every step, from the few clusters that run
// at once; the step kernels store them from all SMs.  16 steps of 14,000 sites x 32
// columns of five entries a row take 0.22 ms against 0.28 in complex128 and 0.21
// against 0.28 in complex64, x 64 0.39 against 0.38 and 0.38 against 0.36, x 128 0.73
// against 0.63 and 0.69 against 0.53; with rows of more than five complex128 entries
// 4,096 x 64 takes 0.24 against 0.27 and x 128 0.39 against 0.32.
template <class T> int chain_plan(int64_t n, int width, int64_t b, ClusterPlan *out) {
    const int64_t most = sizeof(T) == 8 && width > 5 ? 500000 : 850000;
    if (n * b > most) {
        *out = ClusterPlan{};
        return KMSD_OK;
    }
    return find_plan<T>(kChain, n, width, b, out);
}

template <class T>
int cluster_chain(const ClusterPlan &pl, const CsrView<T> &H, int width, int64_t n, const double2 *cur, const double2 *prev,
                  double2 *store, int ring, int64_t b, int64_t k0, int64_t k1, double center, double half, cudaStream_t s) {
    ChainArgs<T> a{H, cur, prev, store, n, b, ring, pl.cols, k0, k1, center, half};
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    cluster_config(cfg, at, pl.groups * pl.size, pl.size, pl.threads, pl.smem);
    cfg.stream = s;
    void *args[] = {&a};
    KMSD_CUDA(cudaLaunchKernelExC(&cfg, pick_chain<T>(width, pl.rpt), args));
    count_launch();
    return KMSD_OK;
}

template <class T>
int cluster_series(const ClusterPlan &pl, const CsrView<T> &H, int width, int64_t n, const T *vim, double wi,
                   const double2 *B, double2 *out, int64_t b, int64_t nb, int64_t phi0, bool write_psi,
                   const double *coeff, int64_t ncoeff, double center, double half, int *status, cudaStream_t s) {
    SeriesArgs<T> a;
    std::memset(&a, 0, sizeof(a));
    a.H = H;
    a.vim = vim;
    a.B = B;
    a.out = out;
    a.n = n;
    a.b = b;
    a.nb = nb;
    a.phi0 = phi0;
    a.write_psi = write_psi;
    a.cols = pl.cols;
    a.terms = (int)ncoeff;
    a.center = center;
    a.half = half;
    a.wi = (T)wi;
    a.status = status;
    for (int64_t i = 0; i < 2 * ncoeff; ++i) a.coeff[i] = (T)coeff[i];
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    cluster_config(cfg, at, pl.groups * pl.size, pl.size, pl.threads, pl.smem);
    cfg.stream = s;
    void *args[] = {&a};
    KMSD_CUDA(cudaLaunchKernelExC(&cfg, pick_kernel<T>(width, pl.rpt, vim != nullptr), args));
    count_launch();
    return KMSD_OK;
}

#define KMSD_SERIES_INSTANCES(T)                                                                                        \
    template int series_plan<T>(int64_t, int, int64_t, bool, ClusterPlan *);                                           \
    template int chain_plan<T>(int64_t, int, int64_t, ClusterPlan *);                                                  \
    template int cluster_chain<T>(const ClusterPlan &, const CsrView<T> &, int, int64_t, const double2 *,              \
                                  const double2 *, double2 *, int, int64_t, int64_t, int64_t, double, double,          \
                                  cudaStream_t);                                                                       \
    template int cluster_series<T>(const ClusterPlan &, const CsrView<T> &, int, int64_t, const T *, double,           \
                                   const double2 *, double2 *, int64_t, int64_t, int64_t, bool, const double *,        \
                                   int64_t, double, double, int *, cudaStream_t);
KMSD_SERIES_INSTANCES(double)
KMSD_SERIES_INSTANCES(float)
#undef KMSD_SERIES_INSTANCES

}  // namespace kmsd
