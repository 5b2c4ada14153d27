// Chebyshev moments of small orthogonal-basis operators in ONE launch.
//
// One step of a small lattice (4,096 sites, 8 vectors: 0.5 MB per vector block)
// is a few microseconds of kernel, most of it launch, ramp and tail, and there
// are hundreds of steps in a call.  The columns of the recurrence never meet, so
// a thread-block cluster takes a few columns through ALL steps: its CTAs share
// out the rows, T_k and T_{k-1} stay in their shared memory, a thread keeps the
// entries of its rows (column addresses and values) in registers, neighbours on
// another CTA are read through distributed shared memory, and the CTAs meet at
// the cluster's hardware barrier once per step (about 0.2 us).  The column sums
// of a step are reduced in the warp, then by a warp of its own during the next
// step, and leave shared memory every kHist steps, so that no global store
// stands before the barrier.
//
// What bounds it: for few columns the latency of one row's chain (loads, 2W
// fused multiply-adds, store) and the meeting, 0.8-1 us a step; for many, the
// shared-memory traffic, (W + 3) elements per row and column.  A cluster of up to
// 16 CTAs whose threads own up to 4 rows covers about 30,000 rows.  M = 512
// direct moments of 4,096 sites x 8 complex128 columns took 0.55 ms against 4.33
// with a launch per step; 511 of 16,129 x 31 complex64 by the product identity
// 0.89 ms against 5.39.  Within its reach it was the faster one everywhere: from
// 512 to 30,720 rows and 1 to 256 columns by 1.5 (28,900 x 256) to 10 times.
//
// The arithmetic of an element is that of cheb_step_kernel, entry by entry, so
// complex64 vectors come out bit-identical; the FP64 sums are taken in another
// (fixed) order.
#include <algorithm>
#include <cstring>
#include <map>
#include <mutex>
#include <tuple>

#include "kmsd_cluster.cuh"

using namespace kmsd;

namespace {

constexpr int kHist = 64;        // steps whose sums are held in shared memory
// Threads that own rows (one more warp sums): what 96 (complex64) or 128
// (complex128) registers a thread allow.
template <class T> constexpr int kMaxCompute = sizeof(T) == 4 ? 608 : 480;

template <class T> struct Cx;
template <> struct Cx<double> { using type = double2; };
template <> struct Cx<float> { using type = float2; };

template <class T> struct ClusterArgs {
    CsrView<T> H;
    const double2 *B;
    int64_t b;
    const ClusterSystem *systems;  // nullptr: one
    ClusterSystem one;
    int groups, cols, rows;
    int64_t length;
    int steps;
    double *partial;  // [cluster][step][CTA][2 * cols]
};

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
// An element from any CTA's shared memory.
__device__ __forceinline__ double2 load_far(unsigned at, double2) {
    double2 v;
    asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(at));
    return v;
}
__device__ __forceinline__ float2 load_far(unsigned at, float2) {
    float2 v;
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(at));
    return v;
}

// Sums NV values over the lanes of a warp; the lane whose low bits are zero
// returns true and holds the sum of value `which` in v[0].  Halving the values
// with every exchange takes NV - 1 + log2(32 / NV) exchanges instead of 5 NV.
template <int NV>
__device__ __forceinline__ bool warp_sums(double (&v)[NV], int lane, int &which) {
    which = 0;
    int off = 16;
#pragma unroll
    for (int h = NV / 2; h >= 1; h /= 2, off /= 2) {
        const bool up = lane & off;
#pragma unroll
        for (int i = 0; i < h; ++i) {
            const double give = up ? v[i] : v[i + h], keep = up ? v[i + h] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, give, off);
        }
        if (up) which += h;
    }
    const int rest = 2 * off - 1;
    for (; off > 0; off /= 2) v[0] += __shfl_xor_sync(0xffffffffu, v[0], off);
    return (lane & rest) == 0;
}

// Rows of up to W entries, RPT rows per thread, CG columns at a time.
template <class T, bool DIRECT, int W, int RPT, int CG>
__global__ void __launch_bounds__(kMaxCompute<T> + 32, 1) cluster_moments_kernel(const ClusterArgs<T> a) {
    using V = typename Cx<T>::type;
    constexpr int NS = DIRECT ? 1 : 2;  // sums per column
    extern __shared__ __align__(16) unsigned char sm[];
    unsigned rank, size;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(size));
    const int cluster = blockIdx.x / size;
    const ClusterSystem sys = a.systems ? a.systems[cluster / a.groups] : a.one;
    const int c0 = (cluster % a.groups) * a.cols;
    const int cols = min(a.cols, (int)(a.b - c0));
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int compute = blockDim.x - 32, warps = compute / 32;
    const int rows = a.rows;
    const int mine = max(0, min(rows, (int)(sys.n - (int64_t)rank * rows)));
    const unsigned plane = (unsigned)rows * sizeof(V), block = plane * a.cols;
    const unsigned base = (unsigned)__cvta_generic_to_shared(sm);
    // [T_k | T_{k-1} (| bra)][column][row], the sums of the warps (two steps), the history
    V *vec = reinterpret_cast<V *>(sm);
    const size_t vec_bytes = ((size_t)block * (DIRECT ? 3 : 2) + 15) / 16 * 16;
    double *red = reinterpret_cast<double *>(sm + vec_bytes);
    const int nv = NS * a.cols;
    double *hist = red + 4 * warps * nv;

    // ---- this thread's rows: where each entry's column lies and its value
    // (short rows read their own element times zero)
    unsigned at[RPT][W];
    T val[RPT][W];
    bool far[RPT];  // a row of this warp has a column on another CTA
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
        const int r = i * compute + tid;
        const bool on = tid < compute && r < mine;
        const int64_t g = sys.row0 + (int64_t)rank * rows + r;
        const int k0 = on ? a.H.ptr[g] : 0, k1 = on ? a.H.ptr[g + 1] : 0;
        bool away = false;
#pragma unroll
        for (int j = 0; j < W; ++j) {
            at[i][j] = base + (on ? (unsigned)r * (unsigned)sizeof(V) : 0u);
            val[i][j] = T(0);
            if (k0 + j < k1) {
                const int rel = (int)(a.H.idx[k0 + j] - sys.row0), owner = rel / rows, loc = rel - owner * rows;
                val[i][j] = a.H.re[k0 + j];
                at[i][j] = base + (unsigned)loc * (unsigned)sizeof(V);
                if (owner != (int)rank) {
                    at[i][j] = remote_address(at[i][j], owner);
                    away = true;
                }
            }
        }
        far[i] = __any_sync(0xffffffffu, away);
    }
    for (int i = tid; i < mine * cols; i += blockDim.x) {
        const int r = i / cols, c = i - r * cols;
        const double2 v = a.B[(sys.row0 + (int64_t)rank * rows + r) * a.b + c0 + c];
        V w;
        w.x = (T)v.x;
        w.y = (T)v.y;
        vec[(size_t)c * rows + r] = w;
        if (DIRECT) vec[(size_t)(2 * a.cols + c) * rows + r] = w;
        w.x = w.y = T(0);
        vec[(size_t)(a.cols + c) * rows + r] = w;  // "T_{-1}": the first step is t - 0
    }
    cluster_sync_all();

    const T cen = (T)sys.center, hal = (T)sys.half, inv = (T)(1. / sys.half);
    double *out = a.partial + (size_t)cluster * (a.steps + (DIRECT ? 1 : 0)) * size * nv;
    // Sums of a step over the warps, by the last warp; full histories leave.
    auto collect = [&](int k, bool last) {
        const double *src = red + (k & 3) * warps * nv;
        for (int v = lane; v < nv; v += 32) {
            double s = 0.;
            for (int w = 0; w < warps; ++w) s += src[w * nv + v];
            hist[(k % kHist) * nv + v] = s;
        }
        if (k % kHist == kHist - 1 || last) {
            __syncwarp();
            const int first = k / kHist * kHist;
            for (int i = lane; i < (k - first + 1) * nv; i += 32) {
                const int kk = i / nv, v = i - kk * nv;
                out[((size_t)(first + kk) * size + rank) * nv + v] = hist[i];
            }
        }
    };
    // The sums of CG columns from c on, over the warp, for step `sum`.
    auto put = [&](double (&s)[NS * CG], int c, int sum) {
        int which;
        if (warp_sums<NS * CG>(s, lane, which) && c + which / NS < cols)
            red[((sum & 3) * warps + warp) * nv + c * NS + which] = s[0];
    };
    // DIRECT: sum 0 is <B, B>, sum k is <B, T_k>; else sum k - 1 holds <T_{k-1}, T_{k-1}> and <T_{k-1}, T_k>
    int sums = 0;
    if (DIRECT) {
        if (tid < compute)
            for (int c = 0; c < cols; c += CG) {
                double s[NS * CG];
#pragma unroll
                for (int q = 0; q < NS * CG; ++q) {
                    s[q] = 0.;
                    if (c + q < cols)
                        for (int r = tid; r < mine; r += compute) {
                            const V x = vec[(size_t)(c + q) * rows + r];
                            s[q] += (double)x.x * (double)x.x + (double)x.y * (double)x.y;
                        }
                }
                put(s, c, 0);
            }
        sums = 1;
        cluster_sync_all();
    }
    unsigned cur = 0;  // offset of T_{k-1}; T_k goes to the other block, over T_{k-2}
    T two = T(1);      // 2, and 1 in the first step
    for (int k = 1; k <= a.steps; ++k) {
        if (tid < compute) {
            const unsigned nxt = block - cur;
            for (int c = 0; c < cols; c += CG) {
                double s[NS * CG];
#pragma unroll
                for (int q = 0; q < NS * CG; ++q) s[q] = 0.;
#pragma unroll
                for (int q = 0; q < CG; ++q) {
                    if (CG == 1 || c + q < cols) {
                        const unsigned off = (unsigned)(c + q) * plane, from = off + cur;
#pragma unroll
                        for (int i = 0; i < RPT; ++i) {
                            const int r = i * compute + tid;
                            if (RPT == 1 || i == 0 || r < mine) {  // (idle lanes of the first row repeat row 0's reads)
                                const unsigned me = off + (unsigned)(r < mine ? r : 0) * (unsigned)sizeof(V);
                                V xv[W];
                                if (far[i]) {
#pragma unroll
                                    for (int j = 0; j < W; ++j) xv[j] = load_far(at[i][j] + from, V{});
                                } else {
#pragma unroll
                                    for (int j = 0; j < W; ++j)
                                        xv[j] = *reinterpret_cast<const V *>(sm + (at[i][j] + from - base));
                                }
                                const V x = *reinterpret_cast<const V *>(sm + me + cur);
                                V *dst = reinterpret_cast<V *>(sm + me + nxt);
                                const V pv = *dst;  // T_{k-2}
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
                                if (r < mine) {
                                    *dst = nx;
                                    if (DIRECT) {
                                        const V br = *reinterpret_cast<const V *>(sm + me + 2 * block);
                                        s[q] += (double)br.x * (double)nx.x + (double)br.y * (double)nx.y;
                                    } else {
                                        doubling_sums<T>(s[2 * q], s[2 * q + (DIRECT ? 0 : 1)], x.x, x.y, nx.x, nx.y);
                                    }
                                }
                            }
                        }
                    }
                }
                if (c + CG >= cols) cluster_arrive();  // T_k is written: its sums overlap the meeting
                put(s, c, sums);
            }
        } else {
            cluster_arrive();
            if (sums > 1) collect(sums - 2, false);  // written before the last meeting
        }
        cluster_wait();
        ++sums;
        cur = block - cur;
        two = T(2);
    }
    cluster_sync_all();
    if (tid >= compute) {
        if (sums > 1) collect(sums - 2, false);
        collect(sums - 1, true);
    }
    cluster_sync_all();
    // ---- moments: the CTAs share out the steps
    auto total = [&](int k, int v) {
        double s = 0.;
        for (unsigned q = 0; q < size; ++q) s += __ldcg(out + ((size_t)k * size + q) * nv + v);
        return s;
    };
    for (int i = (int)rank * blockDim.x + tid; i < sums * cols; i += (int)size * blockDim.x) {
        const int k = i / cols, c = i - k * cols;
        double *mu = sys.mu + c0 + c;
        if (DIRECT) {
            mu[(size_t)k * a.b] = total(k, c);
        } else {
            const double se = total(k, 2 * c), so = total(k, 2 * c + 1);
            if (k == 0) {
                mu[0] = se;
                if (a.length > 1) mu[a.b] = so;
            } else {
                const double mu0 = total(0, 2 * c), mu1 = total(0, 2 * c + 1);
                if (2 * k < a.length) mu[(size_t)(2 * k) * a.b] = 2. * se - mu0;
                if (2 * k + 1 < a.length) mu[(size_t)(2 * k + 1) * a.b] = 2. * so - mu1;
            }
        }
    }
}

template <class T, bool DIRECT, int W>
const void *pick_shape(int rpt, int cg) {
    switch (rpt) {
        case 1:
            return cg == 1 ? (const void *)cluster_moments_kernel<T, DIRECT, W, 1, 1>
                           : (const void *)cluster_moments_kernel<T, DIRECT, W, 1, 4>;
        case 2:
            return cg == 1 ? (const void *)cluster_moments_kernel<T, DIRECT, W, 2, 1>
                           : (const void *)cluster_moments_kernel<T, DIRECT, W, 2, 4>;
    }
    if constexpr (W < kClusterWidth)
        return cg == 1 ? (const void *)cluster_moments_kernel<T, DIRECT, W, 4, 1>
                       : (const void *)cluster_moments_kernel<T, DIRECT, W, 4, 4>;
    return nullptr;
}
// Rows a thread may own: the entries of four rows of eight do not fit its registers.
int most_rows(int width) { return width < 6 ? 4 : 2; }
template <class T>
const void *pick_kernel(bool direct, int width, int rpt, int cg) {
    if (width <= 4) return direct ? pick_shape<T, true, 4>(rpt, cg) : pick_shape<T, false, 4>(rpt, cg);
    if (width <= 5) return direct ? pick_shape<T, true, 5>(rpt, cg) : pick_shape<T, false, 5>(rpt, cg);
    return direct ? pick_shape<T, true, 8>(rpt, cg) : pick_shape<T, false, 8>(rpt, cg);
}

// Dynamic shared memory a CTA may have on this device.
size_t smem_limit() {
    static const size_t limit = [] {
        int dev = 0, optin = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        return (size_t)optin - 1024;
    }();
    return limit;
}

void cluster_config(cudaLaunchConfig_t &cfg, cudaLaunchAttribute *at, int ctas, int size, int threads, size_t smem) {
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = size;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
}

// Clusters of this shape that run at once (cached; also sets the kernel's
// attributes on first use).
int active_clusters(const void *kernel, int size, int threads, size_t smem) {
    static std::mutex lock;
    static std::map<std::tuple<const void *, int, int, size_t>, int> cache;
    std::lock_guard<std::mutex> guard(lock);
    const auto key = std::make_tuple(kernel, size, threads, smem);
    auto it = cache.find(key);
    if (it != cache.end()) return it->second;
    int n = 0;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    cluster_config(cfg, at, size, size, threads, smem);
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_limit()) != cudaSuccess ||
        cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
        cudaGetLastError();
        n = 0;
    }
    if (cache.size() >= 4096) cache.clear();
    cache[key] = n;
    return n;
}

}  // namespace

namespace kmsd {

template <class T>
int cluster_plan(int64_t n, int width, int64_t b, bool doubling, int64_t systems, ClusterPlan *out) {
    *out = ClusterPlan{};
    if (width < 1 || width > kClusterWidth) return KMSD_OK;
    static std::mutex lock;
    static std::map<std::tuple<int64_t, int, int64_t, bool, int64_t>, ClusterPlan> cache;
    const auto key = std::make_tuple(n, width, b, doubling, systems);
    {
        std::lock_guard<std::mutex> guard(lock);
        const auto it = cache.find(key);
        if (it != cache.end()) {
            *out = it->second;
            return KMSD_OK;
        }
    }
    const int elem = 2 * sizeof(T), blocks = doubling ? 2 : 3, ns = doubling ? 2 : 1;
    double best = 0.;
    for (int size : {16, 8, 4, 2, 1}) {
        const int64_t rows = (n + size - 1) / size;
        if (rows > most_rows(width) * kMaxCompute<T>) continue;
        const int rpt = rows <= kMaxCompute<T> ? 1 : rows <= 2 * kMaxCompute<T> ? 2 : 4;
        const int compute = (int)(((rows + rpt - 1) / rpt + 31) / 32 * 32), threads = compute + 32;
        for (int cols = 1; cols <= std::min<int64_t>(b, 32); ++cols) {
            const int cg = cols == 1 ? 1 : 4;
            const size_t vec = ((size_t)rows * cols * elem * blocks + 15) / 16 * 16;
            const size_t smem = vec + (size_t)(4 * (compute / 32) + kHist) * ns * cols * 8;
            if (smem > smem_limit()) break;
            const int64_t groups = (b + cols - 1) / cols;
            const int act = active_clusters(pick_kernel<T>(!doubling, width, rpt, cg), size, threads, smem);
            if (act < 1) continue;
            const int64_t waves = (groups * systems + act - 1) / act;
            // cycles of a step: the chain of one row and the meeting, then the
            // shared-memory traffic (fitted to 0.8 us for 64 rows x 1 column of a
            // CTA and 3.1 us for 1009 x 5 complex64)
            const double step = (size > 1 ? 1300. : 900.) + (double)rows * cols * (width + (doubling ? 3 : 4)) * elem / 75.;
            const double cost = step * waves;
            if (out->size == 0 || cost < best) {
                best = cost;
                *out = ClusterPlan{size, (int)rows, cols, (int)groups, rpt, threads, cg, smem};
            }
        }
    }
    std::lock_guard<std::mutex> guard(lock);
    if (cache.size() >= 1024) cache.clear();
    cache[key] = *out;
    return KMSD_OK;
}

size_t cluster_scratch(const ClusterPlan &pl, int64_t systems, int64_t length, bool doubling) {
    const int64_t sums = doubling ? (length + 1) / 2 : length;
    return (size_t)pl.groups * systems * sums * pl.size * (doubling ? 2 : 1) * pl.cols * sizeof(double);
}

template <class T>
int cluster_moments(const ClusterPlan &pl, const CsrView<T> &H, int width, const double2 *B, int64_t b, int64_t length,
                    bool doubling, const ClusterSystem *systems, int64_t count, const ClusterSystem &one, double *scratch,
                    cudaStream_t s) {
    ClusterArgs<T> a;
    std::memset(&a, 0, sizeof(a));
    a.H = H;
    a.B = B;
    a.b = b;
    a.systems = systems;
    a.one = one;
    a.groups = pl.groups;
    a.cols = pl.cols;
    a.rows = pl.rows;
    a.length = length;
    a.steps = (int)(doubling ? (length + 1) / 2 : length - 1);
    a.partial = scratch;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    cluster_config(cfg, at, (int)(pl.groups * count) * pl.size, pl.size, pl.threads, pl.smem);
    cfg.stream = s;
    void *args[] = {&a};
    KMSD_CUDA(cudaLaunchKernelExC(&cfg, pick_kernel<T>(!doubling, width, pl.rpt, pl.cg), args));
    count_launch();
    return KMSD_OK;
}

template int cluster_plan<double>(int64_t, int, int64_t, bool, int64_t, ClusterPlan *);
template int cluster_plan<float>(int64_t, int, int64_t, bool, int64_t, ClusterPlan *);
template int cluster_moments<double>(const ClusterPlan &, const CsrView<double> &, int, const double2 *, int64_t, int64_t, bool,
                                     const ClusterSystem *, int64_t, const ClusterSystem &, double *, cudaStream_t);
template int cluster_moments<float>(const ClusterPlan &, const CsrView<float> &, int, const double2 *, int64_t, int64_t, bool,
                                    const ClusterSystem *, int64_t, const ClusterSystem &, double *, cudaStream_t);

}  // namespace kmsd
