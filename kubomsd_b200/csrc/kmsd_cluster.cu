// Chebyshev moments of small orthogonal-basis operators in ONE launch.
//
// One step of a small lattice (4,096 sites, 8 vectors: 0.5 MB per vector block)
// is a few microseconds of kernel, most of it launch, ramp and tail, and there
// are hundreds of steps in a call.  The columns of the recurrence never meet, so
// a thread-block cluster takes a few columns through ALL steps: its CTAs share
// out the rows, T_k and T_{k-1} stay in their shared memory, a thread keeps the
// entries of its rows (column addresses and values) in registers, neighbours on
// another CTA are read through distributed shared memory, and the CTAs meet at
// the cluster's hardware barrier once per step (about 0.2 us).  Small systems
// share out the columns over the warps too.  The column sums
// of a step are reduced in the warp, then by a warp of its own during the next
// step, and leave shared memory every kHist steps, so that no global store
// stands before the barrier.
//
// What bounds it: for few columns the latency of one row's chain (loads, 2W
// fused multiply-adds, store) and the meeting, 0.8-1 us a step; for many, the
// shared-memory traffic, (W + 3) elements per row and column.  A cluster of up to
// 16 CTAs whose threads own up to 4 rows covers about 30,000 rows.  M = 512
// direct moments of 4,096 sites x 8 complex128 columns take 0.46 ms against 4.33
// with a launch per step; 511 of 16,129 x 31 complex64 by the product identity
// 0.75 ms against 5.38; 256 of 24 lattices of 576 to 25,600 sites x 16 complex64
// in one launch 2.29 ms against 9.00.  Within its reach it is the faster one
// everywhere: from 1,000 to 36,000 rows of 3 to 7 entries and 2 to 128 columns by 1.3
// (9,000 rows of 7 x 128, direct: 1.22 ms against 1.54) to 17 times.
//
// The arithmetic of an element is that of cheb_step_kernel, entry by entry, so
// complex64 vectors come out bit-identical; the FP64 sums are taken in another
// (fixed) order.
#include <algorithm>
#include <cstring>
#include <functional>
#include <map>
#include <mutex>
#include <tuple>
#include <utility>

#include "kmsd_cluster.cuh"

using namespace kmsd;

namespace {

constexpr int kHist = 64;        // steps whose sums are held in shared memory
template <class T> struct ClusterArgs {
    CsrView<T> H;
    const double2 *B;
    int64_t b;
    const ClusterSystem *systems;  // nullptr: `one`, its columns in groups of `cols`
    const ClusterJob *jobs;        // per cluster, with `systems`
    ClusterSystem one;
    int cols;  // most columns of a cluster
    int64_t length;
    int steps;
    double *partial;  // [cluster][step][CTA][2 * cols]
};

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
    ClusterSystem sys = a.one;
    int c0 = cluster * a.cols, cols = min(a.cols, (int)(a.b - c0));
    if (a.systems) {
        const ClusterJob job = a.jobs[cluster];
        sys = a.systems[job.system];
        c0 = job.c0;
        cols = job.cols;
    }
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int compute = blockDim.x - 32;
    const int rows = (int)((sys.n + size - 1) / size);
    const int mine = max(0, min(rows, (int)(sys.n - (int64_t)rank * rows)));
    // Where the rows take at most half of the warps, sets of warps share out the
    // columns: warp w is warp `own` of set w / wr.
    const int cwarps = compute / 32, wr = max(1, (rows + 31) / 32), sets = column_sets(cwarps, rows);
    const int set = sets > 1 ? warp / wr : 0, own = sets > 1 ? warp - set * wr : warp;
    const int at_row = own * 32 + lane;  // this thread's first row; the next ones follow `compute` apart
    const int warps = min(cwarps, (mine + 31) / 32);  // of a set that own rows
    const bool works = warp < cwarps && set < sets && own < warps && set * CG < cols;
    const unsigned plane = (unsigned)rows * sizeof(V), block = plane * cols;
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
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
        const int r = i * compute + at_row;
        const bool on = works && r < mine;
        const int64_t g = sys.row0 + (int64_t)rank * rows + r;
        const int k0 = on ? a.H.ptr[g] : 0, k1 = on ? a.H.ptr[g + 1] : 0;
#pragma unroll
        for (int j = 0; j < W; ++j) {
            at[i][j] = base + (on ? (unsigned)r * (unsigned)sizeof(V) : 0u);
            val[i][j] = T(0);
            if (k0 + j < k1) {
                const int rel = (int)(a.H.idx[k0 + j] - sys.row0), owner = rel / rows, loc = rel - owner * rows;
                val[i][j] = a.H.re[k0 + j];
                at[i][j] = base + (unsigned)loc * (unsigned)sizeof(V);
                if (owner != (int)rank) at[i][j] = remote_address(at[i][j], owner);
            }
        }
    }
    for (int i = tid; i < mine * cols; i += blockDim.x) {
        const int r = i / cols, c = i - r * cols;
        const double2 v = a.B[(sys.row0 + (int64_t)rank * rows + r) * a.b + c0 + c];
        V w;
        w.x = (T)v.x;
        w.y = (T)v.y;
        vec[(size_t)c * rows + r] = w;
        if (DIRECT) vec[(size_t)(2 * cols + c) * rows + r] = w;
        w.x = w.y = T(0);
        vec[(size_t)(cols + c) * rows + r] = w;  // "T_{-1}": the first step is t - 0
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
            __syncwarp();  // the next sums go over this history; no meeting orders the lanes of this warp
        }
    };
    // The sums of CG columns from c on, over the warp, for step `sum`.
    auto put = [&](double (&s)[NS * CG], int c, int sum) {
        int which;
        if (warp_sums<NS * CG>(s, lane, which) && c + which / NS < cols)
            red[((sum & 3) * warps + own) * nv + c * NS + which] = s[0];
    };
    // DIRECT: sum 0 is <B, B>, sum k is <B, T_k>; else sum k - 1 holds <T_{k-1}, T_{k-1}> and <T_{k-1}, T_k>
    int sums = 0;
    if (DIRECT) {
        if (works)
            for (int c = set * CG; c < cols; c += sets * CG) {
                double s[NS * CG];
#pragma unroll
                for (int q = 0; q < NS * CG; ++q) {
                    s[q] = 0.;
                    if (c + q < cols)
                        for (int r = at_row; r < mine; r += compute) {
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
        if (works) {
            const unsigned nxt = block - cur;
            for (int c = set * CG; c < cols; c += sets * CG) {
                double s[NS * CG];
#pragma unroll
                for (int q = 0; q < NS * CG; ++q) s[q] = 0.;
#pragma unroll
                for (int q = 0; q < CG; ++q) {
                    if (CG == 1 || c + q < cols) {
                        const unsigned off = (unsigned)(c + q) * plane, from = off + cur;
#pragma unroll
                        for (int i = 0; i < RPT; ++i) {
                            const int r = i * compute + at_row;
                            if (RPT == 1 || i == 0 || r < mine) {  // (idle lanes of the first row repeat row 0's reads)
                                const unsigned me = off + (unsigned)(r < mine ? r : 0) * (unsigned)sizeof(V);
                                V xv[W];
#pragma unroll
                                for (int j = 0; j < W; ++j) xv[j] = load_any(at[i][j] + from, V{});
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
                if (c + sets * CG >= cols) cluster_arrive();  // T_k is written: its sums overlap the meeting
                put(s, c, sums);
            }
        } else {
            cluster_arrive();
            if (tid >= compute && sums > 1) collect(sums - 2, false);  // written before the last meeting
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
    if constexpr (W < kClusterWidth) {
        if (rpt == 3)
            return cg == 1 ? (const void *)cluster_moments_kernel<T, DIRECT, W, 3, 1>
                           : (const void *)cluster_moments_kernel<T, DIRECT, W, 3, 4>;
        return cg == 1 ? (const void *)cluster_moments_kernel<T, DIRECT, W, 4, 1>
                       : (const void *)cluster_moments_kernel<T, DIRECT, W, 4, 4>;
    }
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

template <class T> int rows_per_thread(int64_t rows) { return (int)((rows + kMaxCompute<T> - 1) / kMaxCompute<T>); }
int cluster_threads(int64_t rows, int rpt) { return (int)(((rows + rpt - 1) / rpt + 31) / 32 * 32) + 32; }
// Shared memory of the vector blocks, and of the sums of a CTA.
template <class T> size_t vec_bytes(int64_t rows, int cols, bool doubling) {
    return ((size_t)rows * cols * 2 * sizeof(T) * (doubling ? 2 : 3) + 15) / 16 * 16;
}
size_t sum_bytes(int threads, int cols, bool doubling) {
    return (size_t)(4 * (threads / 32 - 1) + kHist) * (doubling ? 2 : 1) * cols * sizeof(double);
}
// Cycles of a step of a cluster whose CTAs have `threads`: the meeting, then for
// each (row, column) of a thread the chain of its loads and arithmetic, or the
// shared-memory traffic of all warps where that is more (fitted to 0.9 us for
// 256 rows x 1 complex128 column of a CTA and 2.8 us for 1009 x 5 complex64).
template <class T> double step_cycles(int64_t rows, int cols, int width, bool doubling, int size, int threads) {
    const int warps = threads / 32 - 1, sets = column_sets(warps, (int)rows);
    const int64_t items = (cols + sets - 1) / sets * ((rows + 32 * warps - 1) / (32 * warps));
    const int busy = std::min<int64_t>(warps, sets * ((rows + 31) / 32));
    const double traffic = busy * (width + (doubling ? 3. : 4.)) * (2 * sizeof(T)) * 32 / 128.;
    return (size > 1 ? 1000. : 600.) + items * std::max(400., traffic);
}

}  // namespace

namespace kmsd {

size_t cluster_smem_limit() {
    static PerDevice<size_t> limit;
    return limit.get([](int dev) {
        int optin = 0;
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        return (size_t)optin - 1024;
    });
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

int active_clusters(const void *kernel, int size, int threads, size_t smem) {
    static std::mutex lock;
    static std::map<std::tuple<int, const void *, int, int, size_t>, int> cache;
    std::lock_guard<std::mutex> guard(lock);
    const auto key = std::make_tuple(current_device(), kernel, size, threads, smem);
    auto it = cache.find(key);
    if (it != cache.end()) return it->second;
    int n = 0;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    cluster_config(cfg, at, size, size, threads, smem);
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cluster_smem_limit()) != cudaSuccess ||
        cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
        cudaGetLastError();
        n = 0;
    }
    if (cache.size() >= 4096) cache.clear();
    cache[key] = n;
    return n;
}

template <class T>
int cluster_plan(int64_t n, int width, int64_t b, bool doubling, ClusterPlan *out) {
    *out = ClusterPlan{};
    if (width < 1 || width > kClusterWidth) return KMSD_OK;
    static std::mutex lock;
    static std::map<std::tuple<int, int64_t, int, int64_t, bool>, ClusterPlan> cache;
    const auto key = std::make_tuple(current_device(), n, width, b, doubling);
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
        if (rows > most_rows(width) * kMaxCompute<T>) continue;
        const int rpt = rows_per_thread<T>(rows), threads = cluster_threads(rows, rpt);
        for (int cols = 1; cols <= std::min<int64_t>(b, 32); ++cols) {
            const int cg = cols == 1 ? 1 : 4;
            const size_t smem = vec_bytes<T>(rows, cols, doubling) + sum_bytes(threads, cols, doubling);
            if (smem > cluster_smem_limit()) break;
            const int64_t groups = (b + cols - 1) / cols;
            const int act = active_clusters(pick_kernel<T>(!doubling, width, rpt, cg), size, threads, smem);
            if (act < 1) continue;
            const double cost = step_cycles<T>(rows, cols, width, doubling, size, threads) * ((groups + act - 1) / act);
            if (out->size == 0 || cost < best) {
                best = cost;
                *out = ClusterPlan{size, cols, (int)groups, rpt, threads, cg, smem};
            }
        }
    }
    std::lock_guard<std::mutex> guard(lock);
    if (cache.size() >= 1024) cache.clear();
    cache[key] = *out;
    return KMSD_OK;
}

// Systems of several sizes in one launch: a cluster takes as many columns of a
// system as keep its step below a common length, the longest jobs first.  The
// cluster size and that length are the ones with the shortest schedule on the
// clusters that run at once.
template <class T>
int cluster_batch_plan(const std::vector<int64_t> &rows_of, int width, int64_t b, bool doubling, ClusterPlan *out,
                       std::vector<ClusterJob> *jobs) {
    *out = ClusterPlan{};
    if (width < 1 || width > kClusterWidth) return KMSD_OK;
    const int64_t biggest = *std::max_element(rows_of.begin(), rows_of.end());
    double best = 0.;
    for (int size : {16, 8, 4, 2, 1}) {
        const int64_t rows = (biggest + size - 1) / size;
        if (rows > most_rows(width) * kMaxCompute<T>) continue;
        const int rpt = rows_per_thread<T>(rows), threads = cluster_threads(rows, rpt);
        double last = 0.;
        for (int most = 1; most <= std::min<int64_t>(b, 32); ++most) {
            const double length = step_cycles<T>(rows, most, width, doubling, size, threads);
            // columns of each system, and what they need
            std::vector<std::pair<double, ClusterJob>> list;
            size_t vec = 0;
            int cols = 0;
            for (size_t i = 0; i < rows_of.size(); ++i) {
                const int64_t r = (rows_of[i] + size - 1) / size;
                int c = 1;
                while (c < std::min<int64_t>(b, 32) && step_cycles<T>(r, c + 1, width, doubling, size, threads) <= length) ++c;
                const int groups = (int)((b + c - 1) / c);
                c = (int)((b + groups - 1) / groups);
                cols = std::max(cols, c);
                vec = std::max(vec, vec_bytes<T>(r, c, doubling));
                for (int c0 = 0; c0 < b; c0 += c)
                    list.push_back({step_cycles<T>(r, std::min<int>(c, (int)b - c0), width, doubling, size, threads),
                                    ClusterJob{(int)i, c0, std::min<int>(c, (int)b - c0), 0}});
            }
            const size_t smem = vec + sum_bytes(threads, cols, doubling);
            if (smem > cluster_smem_limit()) break;
            const int cg = cols == 1 ? 1 : 4;
            const int act = active_clusters(pick_kernel<T>(!doubling, width, rpt, cg), size, threads, smem);
            if (act < 1) continue;
            std::stable_sort(list.begin(), list.end(), [](const auto &x, const auto &y) { return x.first > y.first; });
            std::vector<double> busy(act, 0.);  // a heap of the clusters' finishing times
            double end = 0.;
            for (const auto &j : list) {
                std::pop_heap(busy.begin(), busy.end(), std::greater<double>());
                busy.back() += j.first;
                end = std::max(end, busy.back());
                std::push_heap(busy.begin(), busy.end(), std::greater<double>());
            }
            if (out->size == 0 || end < best) {
                best = end;
                *out = ClusterPlan{size, cols, (int)list.size(), rpt, threads, cg, smem};
                jobs->clear();
                for (const auto &j : list) jobs->push_back(j.second);
            }
            if (last > 0. && end > 2. * last) break;
            last = end;
        }
    }
    return KMSD_OK;
}

size_t cluster_scratch(const ClusterPlan &pl, int64_t length, bool doubling) {
    const int64_t sums = doubling ? (length + 1) / 2 : length;
    return (size_t)pl.groups * sums * pl.size * (doubling ? 2 : 1) * pl.cols * sizeof(double);
}

template <class T>
int cluster_moments(const ClusterPlan &pl, const CsrView<T> &H, int width, const double2 *B, int64_t b, int64_t length,
                    bool doubling, const ClusterSystem *systems, const ClusterJob *jobs, const ClusterSystem &one,
                    double *scratch, cudaStream_t s) {
    ClusterArgs<T> a;
    std::memset(&a, 0, sizeof(a));
    a.H = H;
    a.B = B;
    a.b = b;
    a.systems = systems;
    a.jobs = jobs;
    a.one = one;
    a.cols = pl.cols;
    a.length = length;
    a.steps = (int)(doubling ? (length + 1) / 2 : length - 1);
    a.partial = scratch;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    cluster_config(cfg, at, pl.groups * pl.size, pl.size, pl.threads, pl.smem);
    cfg.stream = s;
    void *args[] = {&a};
    KMSD_CUDA(cudaLaunchKernelExC(&cfg, pick_kernel<T>(!doubling, width, pl.rpt, pl.cg), args));
    count_launch();
    return KMSD_OK;
}

#define KMSD_CLUSTER_INSTANCES(T)                                                                                       \
    template int cluster_plan<T>(int64_t, int, int64_t, bool, ClusterPlan *);                                           \
    template int cluster_batch_plan<T>(const std::vector<int64_t> &, int, int64_t, bool, ClusterPlan *,                 \
                                       std::vector<ClusterJob> *);                                                      \
    template int cluster_moments<T>(const ClusterPlan &, const CsrView<T> &, int, const double2 *, int64_t, int64_t,    \
                                    bool, const ClusterSystem *, const ClusterJob *, const ClusterSystem &, double *,   \
                                    cudaStream_t);
KMSD_CLUSTER_INSTANCES(double)
KMSD_CLUSTER_INSTANCES(float)
#undef KMSD_CLUSTER_INSTANCES

}  // namespace kmsd
