// The batched PCG solve of an overlap stored as 4x4 blocks as ONE launch.
//
// A solve of the launch sequence (kmsd_metric.cu) takes three kernels per
// iteration, each a few to tens of microseconds, and every vector passes
// through L2 between them.  Here the CTAs stay: a CTA owns a contiguous range
// of 4x4 block rows for the whole solve, keeps that range's S blocks and
// preconditioner blocks in shared memory, and meets the others twice per
// iteration, at the two reductions.
//
// The iteration is the reference's (Metric::solve, cpp/native.cpp:313-452) with
// S p formed by its own recurrence:
//     w = S z,  p = z + beta p,  S p = w + beta S p,   alpha = rz / <p, S p>
//     x += alpha p,  r -= alpha S p,  z = M^-1 r,      beta = rz' / rz
// The only vector that a CTA needs from the others is then z, which is written
// before the second reduction anyway, so the exchange of p and its meeting go.
// A restart (p = z) takes S p = S z afresh, after `interval` iterations at most
// under the fixed policy, so the recurrence carries no more rounding than the
// one of r.  Column state (alpha, beta, thresholds, active flags) is kept by
// every CTA for itself: all of them sum the same partials in the same order and
// come to the same decisions, so nothing is broadcast.
//
// Forms (the S slice of each CTA has to fit its shared memory in all of them):
//   cluster  one cluster of 16 CTAs, for systems of up to 6144 (block row,
//            column) pairs: it meets at the hardware barrier (about 0.2 us,
//            0.9 us behind global stores), leaves the other SMs to other
//            streams, and puts its sums into the shared memory of all CTAs;
//   grid     a cooperative launch of one CTA per SM, up to 56,832 pairs; sums
//            travel as packets (below) and every reduction is a meeting too;
//   stream   the same launch with the work vectors in memory (L2), any columns.
// The first two copy the block columns that a CTA's rows touch (its halo) to
// shared memory once per product and keep x, r, p and S p in registers; what
// bounds them is the shared-memory reads of the product (see product()) and the
// two meetings.  `stream` gathers z through L1; bound by that gather.
//
// Whole solves through kmsd_metric_solve, block-Jacobi, rtol 1e-10, against the
// launch sequence in turn with it (about 72 iterations each):
//   2,048 orbitals x 8 columns (cluster)    0.71 ms, 3.00 ms before
//   6,912 x 12 (grid)                       0.84 ms, 3.09 ms
//   32,000 x 32 (stream)                    4.58 ms, 8.24 ms
//   55,296 x 16 (stream)                    4.54 ms, 9.40 ms
// The cluster form against the grid form: 0.48 and 0.58 ms on 864 x 4, 0.70 and
// 0.72 on 2,048 x 8, 0.63 and 0.61 on 864 x 16, where it takes a ninth of the SMs.
// The grid form against the stream form: 0.84 and 1.23 on 6,912 x 12, 1.53 and 2.17
// on 16,384 x 8.
#include <algorithm>
#include <cfloat>
#include <climits>
#include <cstring>
#include <type_traits>
#include <vector>

#include "kmsd_pcg.cuh"

using namespace kmsd;

namespace {

struct ResArgs {
    BsrView<double> S;
    int b;
    const double2 *B;
    double2 *Y, *y, *r, *z, *p, *sp, *t;
    const double *diag;
    const double2 *minv;  // block inverses (nullptr: diagonal preconditioner)
    int minv_real;
    const int *halo_off, *halo, *local, *self;
    ColPtr c;
    Counters *cnt;
    double rtol, atol, gap_ratio;
    int maxiter, interval, adaptive;
    int *status;
    FailReportFull *fr;
    unsigned *bar;   // [0] arrivals, [1] a wait ran out, [2] sequence base of the packets
    uint4 *packets;  // [2]: [column][CTA][2], then the totals [column][2]
    int lcw, lks, nch;
    int own, blocks, halos;
};

// Shared memory: reduction scratch and boxes, column state, then the CTA's S
// blocks, preconditioner blocks and block pattern, then its halo.
constexpr int kStateDoubles = 8, kStateInts = 4;
constexpr int kAhead = 1;
// Continuations of a solve at most, and how far above its threshold a column's true
// residual may be for one: where roundings move it by more than the threshold, the
// tolerance is not attainable.
constexpr int kMostRedos = 4;
constexpr double kRedoWithin = 2.;
constexpr int kResThreads = 384, kStreamThreads = 512, kClusterCtas = 16;
// 16-byte units from one S block in shared memory to the next: in the resident
// forms one more than its 8, so that lanes on neighbouring blocks read from
// different banks; in the stream form, whose warps read one block at a time, none
// more, which lets shares of up to about 100 block rows of 16 blocks fit.
constexpr int kResidentUnits = 9, kStreamUnits = 8;
__host__ __device__ inline size_t up16(size_t x) { return (x + 15) / 16 * 16; }
size_t state_bytes(int threads, int ncol, bool cluster) {
    return (size_t)(threads / 32) * ncol * 16 + (size_t)ncol * (16 + kStateDoubles * 8 + kStateInts * 4) +
           (cluster ? (size_t)2 * kClusterCtas * ncol * 16 : 0);
}
__host__ __device__ inline size_t slice_bytes(int own, int blocks, bool cplx, int pre_doubles, int halos,
                                                      int units) {
    return (size_t)blocks * units * (cplx ? 32 : 16) + (size_t)own * pre_doubles * 8 +
           up16(((size_t)blocks + 2 * (size_t)own + 1 + halos) * 4);
}

// Longest wait at a meeting of the CTAs, after which the solve gives up and the
// call reports an error.  The CTAs of a cooperative launch begin as SMs come free,
// so the first ones wait for what other streams still run; ten seconds leave room
// for that.  The solves queued behind one that gave up do not wait again.
constexpr unsigned long long kMeetNs = 10000000000ull;

__device__ __forceinline__ unsigned long long clock_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ unsigned load_acquire(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
// Counts the rounds of a wait; true once it has lasted too long or another CTA gave up.
struct Patience {
    unsigned rounds = 0;
    unsigned long long t0 = 0;
    __device__ __forceinline__ bool out(unsigned *bar) {
        if ((++rounds & 1023u) != 0) return false;
        const unsigned long long t = clock_ns();
        if (t0 == 0) t0 = t;
        if (t - t0 <= kMeetNs && load_acquire(bar + 1) == 0) return false;
        atomicExch(bar + 1, 1u);
        return true;
    }
};
// A double as a packet whose 8-byte halves each carry half of it and the
// sequence number: a reader that finds the number in both has the value, so a
// reduction takes one trip through L2 instead of a counter's and the data's.  Each
// half is one 64-bit element of the vector access, so a half is never torn.
__device__ __forceinline__ void packet_store(uint4 *p, double v, unsigned seq) {
    const unsigned long long lo = (unsigned long long)seq << 32 | (unsigned)__double2loint(v),
                             hi = (unsigned long long)seq << 32 | (unsigned)__double2hiint(v);
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(lo), "l"(hi) : "memory");
}
__device__ __forceinline__ uint4 packet_load(const uint4 *p) {
    unsigned long long lo, hi;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(lo), "=l"(hi) : "l"(p) : "memory");
    return make_uint4((unsigned)lo, (unsigned)(lo >> 32), (unsigned)hi, (unsigned)(hi >> 32));
}
__device__ __forceinline__ double packet_value(const uint4 &v) { return __hiloint2double((int)v.z, (int)v.x); }
__device__ __forceinline__ void copy16(void *smem, const void *global) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(global) : "memory");
}
__device__ __forceinline__ void copies_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void cluster_meet() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

// Sums a column's packets of all CTAs (in one warp) and puts out its total;
// true when a wait ran out.  Not inlined, like totals(): the solve's state
// stays out of their registers.
template <bool MX>
__device__ __noinline__ bool column_total(const uint4 *row, uint4 *out, unsigned seq, unsigned *bar) {
    const int lane = threadIdx.x & 31, ctas = gridDim.x;
    bool late = false;
    double2 s = make_double2(0., 0.);
    constexpr int PER = 5;  // CTAs of a lane taken at once: 160 in one go
    for (int c0 = lane; c0 < ctas; c0 += 32 * PER) {
        uint4 q[PER][2];
        Patience wait;
        while (true) {
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                const int k = min(c0 + 32 * i, ctas - 1);
                q[i][0] = packet_load(row + 2 * k);
                q[i][1] = packet_load(row + 2 * k + 1);
            }
            bool have = true;
#pragma unroll
            for (int i = 0; i < PER; ++i)
                have = have && q[i][0].y == seq && q[i][0].w == seq && q[i][1].y == seq && q[i][1].w == seq;
            if (have || late) break;
            late = wait.out(bar);
        }
#pragma unroll
        for (int i = 0; i < PER; ++i)
            if (c0 + 32 * i < ctas) {
                const double x = packet_value(q[i][0]), y = packet_value(q[i][1]);
                s.x = MX ? fmax(s.x, x) : s.x + x;
                s.y = MX ? fmax(s.y, y) : s.y + y;
            }
    }
    __syncwarp();
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double x = __shfl_xor_sync(0xffffffffu, s.x, o), y = __shfl_xor_sync(0xffffffffu, s.y, o);
        s.x = MX ? fmax(s.x, x) : s.x + x;
        s.y = MX ? fmax(s.y, y) : s.y + y;
    }
    if (lane < 2) packet_store(out + lane, lane ? s.y : s.x, seq);
    return late;
}
// The totals of all columns into tot.
__device__ __noinline__ bool totals(const uint4 *in, double2 *tot, int ncol, unsigned seq, unsigned *bar) {
    bool late = false;
    for (int j = threadIdx.x; j < ncol; j += blockDim.x) {
        uint4 a, b;
        Patience wait;
        while (true) {
            a = packet_load(in + 2 * j);
            b = packet_load(in + 2 * j + 1);
            if ((a.y == seq && a.w == seq && b.y == seq && b.w == seq) || late) break;
            late = wait.out(bar);
        }
        tot[j] = make_double2(packet_value(a), packet_value(b));
    }
    return late;
}

// The two halves of a meeting of a cooperative launch, at a counter: what the CTA
// wrote before (its threads synchronised) is visible to a thread that has waited for
// all arrivals, and to its CTA once that has synchronised.
__device__ __forceinline__ void arrive(unsigned *bar) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
}
// True when the wait ran out.
__device__ __forceinline__ bool wait_for(unsigned *bar, unsigned arrivals) {
    Patience wait;
    while ((int)(load_acquire(bar) - arrivals) < 0)
        if (wait.out(bar)) return true;
    return false;
}
// All CTAs of the solve have arrived, and their writes are visible.  CL: the
// solve is one thread-block cluster and meets at the hardware barrier; else the
// launch is cooperative and meets at a counter, with a bounded wait.
template <bool CL>
__device__ __forceinline__ bool meet(unsigned *bar, unsigned &arrivals) {
    if constexpr (CL) {
        cluster_meet();
        return true;
    } else {
        __syncthreads();
        arrivals += gridDim.x;
        bool late = false;
        if (threadIdx.x == 0) {
            arrive(bar);
            late = wait_for(bar, arrivals);
        }
        return !__syncthreads_or(late);
    }
}

// CL: one cluster; RES: a thread owns one (block row, column) and keeps its
// part of x, r, p, S p in registers, else they live in global memory (L2).
// lcw: log2 of a chunk's columns.
template <int lcw, bool CPLX, bool CL, bool RES>
__global__ void __launch_bounds__(RES ? kResThreads : kStreamThreads, 1) pcg_resident_kernel(const ResArgs a) {
    constexpr int NT = RES ? kResThreads : kStreamThreads, NW = NT / 32, cw = 1 << lcw;
    constexpr int kBlockUnits = RES ? kResidentUnits : kStreamUnits;
    extern __shared__ __align__(16) unsigned char sm[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ks = RES ? 1 << a.lks : 1, nch = RES ? 1 : a.nch, ncol = nch << lcw, b = a.b;
    double2 *red = reinterpret_cast<double2 *>(sm);  // [warp][column]
    double2 *tot = red + NW * ncol;
    double *safe = reinterpret_cast<double *>(tot + ncol);
    double *bn = safe + ncol, *thr = bn + ncol, *rz = thr + ncol, *alpha = rz + ncol, *beta = alpha + ncol,
           *pend = beta + ncol, *rnorm = pend + ncol;
    int *active = reinterpret_cast<int *>(rnorm + ncol);
    int *restart = active + ncol, *brk = restart + ncol, *iters = brk + ncol;
    double2 *box = reinterpret_cast<double2 *>(iters + ncol);  // CL: [2][CTA][column]
    unsigned char *slice = reinterpret_cast<unsigned char *>(box + (CL ? 2 * kClusterCtas * ncol : 0));

    // ---- the CTA's block rows and the thread's place in them
    const int64_t nbr = a.S.nbrows;
    const int64_t I0 = nbr * blockIdx.x / gridDim.x, I1 = nbr * (blockIdx.x + 1) / gridDim.x;
    const int own = (int)(I1 - I0);
    const int col = lane & (cw - 1), part = (lane >> lcw) & (ks - 1);
    const int lsl = RES ? lcw + a.lks : lcw, slot = (warp << (5 - lsl)) + (lane >> lsl), per_pass = NT >> lsl;
    const bool first = part == 0;

    // ---- the CTA's slice of S and of the preconditioner
    const int pre_d = a.minv ? (a.minv_real ? 16 : 32) : 4;
    double2 *vre = reinterpret_cast<double2 *>(slice);
    double2 *vim = vre + (size_t)a.blocks * kBlockUnits;
    double *pre = reinterpret_cast<double *>(CPLX ? vim + (size_t)a.blocks * kBlockUnits : vim);
    int *sidx = reinterpret_cast<int *>(pre + (size_t)a.own * pre_d), *sptr = sidx + a.blocks, *sself = sptr + a.own + 1;
    int *shalo = sself + a.own;  // RES: the halo's block rows
    double2 *stage = reinterpret_cast<double2 *>(slice + slice_bytes(a.own, a.blocks, CPLX, pre_d, RES ? a.halos : 0, kBlockUnits));
    const int nhalo = RES ? a.halo_off[blockIdx.x + 1] - a.halo_off[blockIdx.x] : 0;
    {
        if constexpr (RES) {
            const int *halo = a.halo + a.halo_off[blockIdx.x];
            for (int i = tid; i < nhalo; i += NT) shalo[i] = halo[i];
        }
        const int k0 = a.S.bptr[I0], nk = a.S.bptr[I1] - k0;
        const double2 *gre = reinterpret_cast<const double2 *>(a.S.re) + (size_t)k0 * 8;
        for (int i = tid; i < nk * 8; i += NT) vre[(i >> 3) * kBlockUnits + (i & 7)] = gre[i];
        if (CPLX) {
            const double2 *gim = reinterpret_cast<const double2 *>(a.S.im) + (size_t)k0 * 8;
            for (int i = tid; i < nk * 8; i += NT) vim[(i >> 3) * kBlockUnits + (i & 7)] = gim[i];
        }
        for (int i = tid; i < nk; i += NT) sidx[i] = (RES ? a.local[k0 + i] : a.S.bidx[k0 + i]) << (lcw + 2);
        for (int i = tid; i <= own; i += NT) sptr[i] = a.S.bptr[I0 + i] - k0;
        if constexpr (RES)
            for (int i = tid; i < own; i += NT) sself[i] = a.self[I0 + i] << (lcw + 2);
        for (int i = tid; i < own * pre_d; i += NT) {
            if (a.minv == nullptr) pre[i] = a.diag[4 * I0 + i];
            else if (a.minv_real) pre[i] = a.minv[16 * I0 + i].x;
            else pre[i] = reinterpret_cast<const double *>(a.minv + 16 * I0)[i];
        }
    }
    unsigned base = 0;
    bool gone = false;  // the others gave up before this CTA began, or an earlier solve of the call did
    if constexpr (CL) {
        cluster_meet();  // every CTA of the cluster is running before its boxes are written
    } else {
        base = load_acquire(a.bar + 2);
        gone = __syncthreads_or(load_acquire(a.bar + 1) | load_acquire(reinterpret_cast<unsigned *>(a.status + 3)));
    }

    unsigned arrivals = 0, seq = base;
    int buf = 0;
    using Sum = std::false_type;
    using Max = std::true_type;
    // A chunk's sums over this warp's lanes, for the columns of the chunk.
    auto gather_sums = [&](int ch, double2 v, auto maximum) {
        constexpr bool MX = decltype(maximum)::value;
        for (int o = cw; o < 32; o <<= 1) {
            const double ox = __shfl_xor_sync(0xffffffffu, v.x, o), oy = __shfl_xor_sync(0xffffffffu, v.y, o);
            v.x = MX ? fmax(v.x, ox) : v.x + ox;
            v.y = MX ? fmax(v.y, oy) : v.y + oy;
        }
        if (lane < cw) red[warp * ncol + (ch << lcw) + lane] = v;
    };
    // Column sums over all CTAs into tot (in every CTA), in a fixed order:
    // lanes, warps, CTAs.  Max: the largest value instead.  It is a meeting too:
    // what the CTAs read and wrote before it comes before what any of them reads
    // and writes after it.
    auto reduce = [&](auto maximum) -> bool {
        constexpr bool MX = decltype(maximum)::value;
        auto join = [](double2 &s, double2 q) {
            s.x = MX ? fmax(s.x, q.x) : s.x + q.x;
            s.y = MX ? fmax(s.y, q.y) : s.y + q.y;
        };
        __syncthreads();
        if constexpr (CL) {
            // every CTA puts its sums into the boxes of all
            for (int i = tid; i < kClusterCtas * ncol; i += NT) {
                const int j = i % ncol, dest = i / ncol;
                double2 s = red[j];
#pragma unroll 4
                for (int w = 1; w < NW; ++w) join(s, red[w * ncol + j]);
                unsigned at;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                             : "=r"(at)
                             : "r"((unsigned)__cvta_generic_to_shared(box + ((size_t)buf * kClusterCtas + blockIdx.x) * ncol + j)),
                               "r"(dest));
                asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(at), "d"(s.x), "d"(s.y) : "memory");
            }
            cluster_meet();
            for (int j = warp * 2 + (lane >> 4); j - (lane >> 4) < ncol; j += 2 * NW) {
                double2 s = j < ncol ? box[((size_t)buf * kClusterCtas + (lane & 15)) * ncol + j] : make_double2(0., 0.);
#pragma unroll
                for (int o = 8; o > 0; o >>= 1)
                    join(s, make_double2(__shfl_xor_sync(0xffffffffu, s.x, o), __shfl_xor_sync(0xffffffffu, s.y, o)));
                if ((lane & 15) == 0 && j < ncol) tot[j] = s;
            }
            buf ^= 1;
            __syncthreads();
            return true;
        } else {
            // The totals order nothing but themselves: the CTA that sums a column
            // puts no fence between its reads and its store.  The CTAs meet at the
            // counter besides, in the last warp and in the shadow of the sums, which
            // take a trip more.  (With fences around the packets and in
            // column_total() a solve of 6,912 x 13 took 1.00 ms, with this 0.88.)
            arrivals += gridDim.x;
            if (tid == NT - 1) arrive(a.bar);
            uint4 *all = a.packets + (size_t)buf * ncol * (gridDim.x + 1) * 2, *sums = all + (size_t)ncol * gridDim.x * 2;
            buf ^= 1;
            ++seq;
            for (int j = tid; j < ncol; j += NT) {
                double2 s = red[j];
#pragma unroll 4
                for (int w = 1; w < NW; ++w) join(s, red[w * ncol + j]);
                uint4 *mine = all + ((size_t)j * gridDim.x + blockIdx.x) * 2;
                packet_store(mine, s.x, seq);
                packet_store(mine + 1, s.y, seq);
            }
            // column j is summed in CTA j (mod CTAs), by warp j / CTAs
            bool late = false;
            for (int j = blockIdx.x + warp * gridDim.x; j < ncol; j += NW * gridDim.x)
                late |= column_total<MX>(all + (size_t)j * gridDim.x * 2, sums + 2 * j, seq, a.bar);
            late |= totals(sums, tot, ncol, seq, a.bar);
            if (tid == NT - 1) late |= wait_for(a.bar, arrivals);
            return !__syncthreads_or(late);
        }
    };

    // RES: copies the halo of v to shared memory
    auto fetch = [&](const double2 *v) {
        const int units = nhalo << (lcw + 2);
#pragma unroll 4
        for (int i = tid; i < units; i += NT)
            copy16(stage + i, v + ((size_t)shalo[i >> (lcw + 2)] << (lcw + 2)) + (i & (4 * cw - 1)));
        copies_done();
        __syncthreads();
    };
    // w += (block k of S) x for NC columns
    auto apply = [&](int k, const auto &x, auto &w) {
        constexpr int NC = sizeof(w) / (4 * sizeof(double2));
        const double2 *vr = vre + k * kBlockUnits, *vi = vim + k * kBlockUnits;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const double2 r01 = vr[2 * i], r23 = vr[2 * i + 1];
            const double q[4] = {r01.x, r01.y, r23.x, r23.y};
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    w[c][i].x = fma(q[j], x[c][j].x, w[c][i].x);
                    w[c][i].y = fma(q[j], x[c][j].y, w[c][i].y);
                }
            if (CPLX) {
                const double2 i01 = vi[2 * i], i23 = vi[2 * i + 1];
                const double qi[4] = {i01.x, i01.y, i23.x, i23.y};
#pragma unroll
                for (int j = 0; j < 4; ++j)
#pragma unroll
                    for (int c = 0; c < NC; ++c) {
                        w[c][i].x = fma(-qi[j], x[c][j].y, w[c][i].x);
                        w[c][i].y = fma(qi[j], x[c][j].x, w[c][i].y);
                    }
            }
        }
    };
    // w[i] = sum_k S[4I + i, k] v[k, column] (all parts of the block row
    // summed), v in the staged halo (RES) or in global memory.
    // RES: the reads of shared memory bound it, four cycles for each of the
    // eight 16-byte reads of an S block that serve only the lanes of one
    // column each.  Neighbouring lanes therefore take both of their columns on
    // every second block and hand each other the sums: per block and column 8
    // reads instead of 12.
    auto product = [&](const double2 *v, int ch, int li, bool on, double2 (&w)[4]) {
        const int k0 = on ? sptr[li] : 0, k1 = on ? sptr[li + 1] : 0;
        double2 ww[RES ? 2 : 1][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) ww[0][i] = ww[RES ? 1 : 0][i] = make_double2(0., 0.);
        if constexpr (RES) {
            const int step = 2 * ks;
            for (int k = k0 + 2 * part + (lane & 1); k < k1; k += step) {
                const double2 *xs = stage + sidx[k];
                double2 x[2][4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    x[0][j] = xs[j * cw + col];
                    x[1][j] = xs[j * cw + (col ^ 1)];
                }
                apply(k, x, ww);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                w[i].x = ww[0][i].x + __shfl_xor_sync(0xffffffffu, ww[1][i].x, 1);
                w[i].y = ww[0][i].y + __shfl_xor_sync(0xffffffffu, ww[1][i].y, 1);
            }
            for (int o = cw; o < cw * ks; o <<= 1)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    w[i].x += __shfl_xor_sync(0xffffffffu, w[i].x, o);
                    w[i].y += __shfl_xor_sync(0xffffffffu, w[i].y, o);
                }
        } else {
            // AHEAD blocks' rows are under way while one is applied
            constexpr int AHEAD = kAhead;
            const double2 *vu = v + ((size_t)ch * nbr << (lcw + 2)) + col;
            double2 x[AHEAD + 1][1][4];
#pragma unroll
            for (int d = 0; d < AHEAD; ++d)
                if (k0 + d < k1) {
                    const double2 *xs = vu + sidx[k0 + d];
#pragma unroll
                    for (int j = 0; j < 4; ++j) x[d][0][j] = xs[j * cw];
                }
            for (int k = k0; k < k1; k += AHEAD + 1) {
#pragma unroll
                for (int d = 0; d <= AHEAD; ++d) {
                    if (k + d + AHEAD < k1) {
                        const double2 *xs = vu + sidx[k + d + AHEAD];
#pragma unroll
                        for (int j = 0; j < 4; ++j) x[(d + AHEAD) % (AHEAD + 1)][0][j] = xs[j * cw];
                    }
                    if (k + d < k1) apply(k + d, x[d], ww);
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) w[i] = ww[0][i];
        }
    };
    // z = M^-1 r on one block row (native.cpp:259-277)
    auto precondition = [&](int li, const double2 (&r)[4], double2 (&z)[4]) {
        if (a.minv == nullptr) {
#pragma unroll
            for (int i = 0; i < 4; ++i) z[i] = make_double2(r[i].x / pre[4 * li + i], r[i].y / pre[4 * li + i]);
        } else if (a.minv_real) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                z[i] = make_double2(0., 0.);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const double q = pre[16 * li + 4 * i + k];
                    z[i].x = fma(q, r[k].x, z[i].x);
                    z[i].y = fma(q, r[k].y, z[i].y);
                }
            }
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                z[i] = make_double2(0., 0.);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const double2 q = reinterpret_cast<const double2 *>(pre)[16 * li + 4 * i + k];
                    z[i].x = fma(q.x, r[k].x, fma(-q.y, r[k].y, z[i].x));
                    z[i].y = fma(q.x, r[k].y, fma(q.y, r[k].x, z[i].y));
                }
            }
        }
    };
    // f(li, on, u) for the block rows of this thread in one chunk, u its
    // column; every thread makes the same passes.
    auto rows = [&](int ch, auto &&f) {
        const int u = (ch << lcw) + col;
        if constexpr (RES) {
            f(slot, slot < own, u);
        } else {
            for (int at = 0; at < own; at += per_pass) f(at + slot, at + slot < own, u);
        }
    };
    // row i of block row li in a work vector
    auto at = [&](int ch, int li, int i) { return (((size_t)ch * nbr + I0 + li) * 4 + i << lcw) + col; };
    auto input = [&](int li, int i, int u) {
        return u < b ? a.B[(4 * (I0 + li) + i) * (int64_t)b + u] : make_double2(0., 0.);
    };

    // state of a resident thread
    double2 ys[4], rs[4], ps[4], ss[4];
    if constexpr (RES) {
#pragma unroll
        for (int i = 0; i < 4; ++i) ys[i] = rs[i] = ps[i] = ss[i] = make_double2(0., 0.);
    }

    bool alive = true;  // no wait has run out
    // ---- column scale: max |Re|, |Im|; nonfinite entries (native.cpp:320-329)
    for (int ch = 0; ch < nch; ++ch) {
        double2 m = make_double2(0., 0.);
        rows(ch, [&](int li, bool on, int u) {
            if (on) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const double2 v = input(li, i, u);
                    if (!isfinite(v.x) || !isfinite(v.y)) m.y = 1.;
                    m.x = fmax(m.x, fmax(fabs(v.x), fabs(v.y)));
                }
            }
        });
        gather_sums(ch, m, Max{});
    }
    alive = !gone && reduce(Max{});
    bool nan_in = false;
    for (int j = tid; j < ncol; j += NT) {
        safe[j] = tot[j].x == 0. ? 1. : tot[j].x;
        nan_in |= tot[j].y != 0.;
    }
    const bool nonfinite = __syncthreads_or(nan_in);
    // ---- q = B / safe, r = q, x = 0, z = M^-1 r
    for (int ch = 0; ch < nch; ++ch) {
        double2 acc = make_double2(0., 0.);
        rows(ch, [&](int li, bool on, int u) {
            if (!on) return;
            const double sf = safe[u];
            double2 rr[4], zz[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const double2 v = input(li, i, u);
                rr[i] = make_double2(v.x / sf, v.y / sf);
            }
            precondition(li, rr, zz);
            if constexpr (RES) {
#pragma unroll
                for (int i = 0; i < 4; ++i) rs[i] = rr[i];
            }
            if (first) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const size_t o = at(ch, li, i);
                    a.z[o] = zz[i];
                    if constexpr (!RES) {
                        a.r[o] = rr[i];
                        a.y[o] = make_double2(0., 0.);
                    }
                    acc.x += rr[i].x * rr[i].x + rr[i].y * rr[i].y;
                    acc.y += rr[i].x * zz[i].x + rr[i].y * zz[i].y;
                }
            }
        });
        gather_sums(ch, acc, Sum{});
    }
    alive = alive && reduce(Sum{});
    bool todo = false;
    for (int j = tid; j < ncol; j += NT) {
        bn[j] = sqrt(tot[j].x);
        thr[j] = fmax(a.rtol * bn[j], a.atol / safe[j]);
        const int act = j < b && bn[j] > thr[j];
        active[j] = act;
        rz[j] = tot[j].y;
        restart[j] = 1;  // the first direction is z
        alpha[j] = beta[j] = pend[j] = 0.;
        brk[j] = iters[j] = 0;
        todo |= act != 0;
    }
    int halt = !__syncthreads_or(todo);
    int broken = 0;
    long long checks = 0, restarts = 0;

    // x in memory: the resident one, or with the step alpha p that is left over
    // from the last update
    auto flush = [&]() {
        for (int ch = 0; ch < nch; ++ch)
            rows(ch, [&](int li, bool on, int u) {
                if (!on || !first) return;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const size_t o = at(ch, li, i);
                    if constexpr (RES) {
                        a.y[o] = ys[i];
                    } else {
                        const double al = pend[u];
                        if (al != 0.) {
                            const double2 pv = a.p[o];
                            double2 yv = a.y[o];
                            yv.x = fma(pv.x, al, yv.x);
                            yv.y = fma(pv.y, al, yv.y);
                            a.y[o] = yv;
                        }
                    }
                }
            });
        __syncthreads();
        for (int j = tid; j < ncol; j += NT) pend[j] = 0.;
    };

    int k = 0, redos = 0;
    while (true) {
        bool accept = true;  // the next true residual decides the solve
        while (alive && !halt && !broken && k < a.maxiter) {
            // ---- p = z + beta p, S p = S z + beta S p, <p, S p>
            for (int ch = 0; ch < nch; ++ch) {
                if constexpr (RES) fetch(a.z);
                double2 acc = make_double2(0., 0.);
                rows(ch, [&](int li, bool on, int u) {
                    double2 w[4];
                    product(a.z, ch, li, on, w);
                    if (!on) return;
                    const bool act = active[u], rst = restart[u];
                    const double be = beta[u], al = pend[u];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const size_t o = at(ch, li, i);
                        double2 pv = make_double2(0., 0.), sv = make_double2(0., 0.);
                        if constexpr (RES) {
                            pv = ps[i];
                            sv = ss[i];
                        } else {
                            if (al != 0. || !rst) pv = a.p[o];
                            if (!rst) sv = a.sp[o];
                            if (al != 0. && first) {
                                double2 yv = a.y[o];
                                yv.x = fma(pv.x, al, yv.x);
                                yv.y = fma(pv.y, al, yv.y);
                                a.y[o] = yv;
                            }
                        }
                        const double2 zv = RES ? stage[sself[li] + i * cw + col] : a.z[o];
                        if (!act) {
                            pv = sv = make_double2(0., 0.);
                        } else if (rst) {
                            pv = zv;
                            sv = w[i];
                        } else {
                            pv = make_double2(fma(be, pv.x, zv.x), fma(be, pv.y, zv.y));
                            sv = make_double2(fma(be, sv.x, w[i].x), fma(be, sv.y, w[i].y));
                        }
                        if constexpr (RES) {
                            ps[i] = pv;
                            ss[i] = sv;
                        }
                        if (first) {
                            if constexpr (!RES) {
                                a.p[o] = pv;
                                a.sp[o] = sv;
                            }
                            acc.x += pv.x * sv.x + pv.y * sv.y;
                            acc.y += pv.x * sv.y - pv.y * sv.x;
                        }
                    }
                });
                gather_sums(ch, acc, Sum{});
            }
            if (!(alive = reduce(Sum{}))) break;
            bool bad = false;
            for (int j = tid; j < b; j += NT) {
                const double cr = tot[j].x, ci = tot[j].y;
                const bool act = active[j];
                if (act && (!(cr > 0.) || !isfinite(cr) || !isfinite(ci) || fabs(ci) > 1e-10 * fmax(fabs(cr), DBL_MIN))) {
                    brk[j] = 1;
                    bad = true;
                }
                alpha[j] = act ? rz[j] / cr : 0.;
                pend[j] = 0.;
            }
            if (__syncthreads_or(bad)) {
                broken = 1;
                break;
            }
            // ---- x += alpha p, r -= alpha S p, z = M^-1 r; |r|^2, Re<r, z>
            for (int ch = 0; ch < nch; ++ch) {
                double2 acc = make_double2(0., 0.);
                rows(ch, [&](int li, bool on, int u) {
                    if (!on) return;
                    const double al = alpha[u];
                    double2 rr[4], zz[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const size_t o = at(ch, li, i);
                        if constexpr (RES) {
                            ys[i].x = fma(ps[i].x, al, ys[i].x);
                            ys[i].y = fma(ps[i].y, al, ys[i].y);
                            rs[i].x = fma(-ss[i].x, al, rs[i].x);
                            rs[i].y = fma(-ss[i].y, al, rs[i].y);
                            rr[i] = rs[i];
                        } else {
                            const double2 sv = a.sp[o];
                            rr[i] = a.r[o];
                            rr[i].x = fma(-sv.x, al, rr[i].x);
                            rr[i].y = fma(-sv.y, al, rr[i].y);
                        }
                    }
                    precondition(li, rr, zz);
                    if (first) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const size_t o = at(ch, li, i);
                            a.z[o] = zz[i];
                            if constexpr (!RES) a.r[o] = rr[i];
                            acc.x += rr[i].x * rr[i].x + rr[i].y * rr[i].y;
                            acc.y += rr[i].x * zz[i].x + rr[i].y * zz[i].y;
                        }
                    }
                });
                gather_sums(ch, acc, Sum{});
            }
            if (!(alive = reduce(Sum{}))) break;
            bool cand = false, left = false;
            bool check = (k + 1) % a.interval == 0;
            for (int j = tid; j < b; j += NT) {
                const int act = active[j];
                iters[j] += act;
                rnorm[j] = sqrt(tot[j].x);
                pend[j] = alpha[j];
                cand |= act && rnorm[j] <= thr[j];
            }
            if (a.adaptive) check = __syncthreads_or(cand) || check;
            ++k;
            if (check) {
                accept = false;
                break;
            }
            for (int j = tid; j < b; j += NT) {
                int act = active[j];
                if (!a.adaptive) act = act && rnorm[j] > thr[j];
                active[j] = act;
                restart[j] = 0;
                const double old = rz[j], now = tot[j].y;
                beta[j] = act ? now / (old != 0. ? old : 1.) : 0.;
                rz[j] = now;
                left |= act != 0;
            }
            halt = !__syncthreads_or(left);
        }
        if (!alive) break;
        // ---- true residual t = q - S x: restart decision (native.cpp:379-402) or
        // acceptance (native.cpp:413-423)
        __syncthreads();
        flush();
        if (!(alive = meet<CL>(a.bar, arrivals))) break;
        for (int ch = 0; ch < nch; ++ch) {
            if constexpr (RES) fetch(a.y);
            double2 acc = make_double2(0., 0.);
            rows(ch, [&](int li, bool on, int u) {
                double2 w[4];
                product(a.y, ch, li, on, w);
                if (!on) return;
                const double sf = safe[u];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const size_t o = at(ch, li, i);
                    const double2 v = input(li, i, u);
                    const double2 t = make_double2(v.x / sf - w[i].x, v.y / sf - w[i].y);
                    const double2 rv = RES ? rs[i] : a.r[o];
                    if (first) {
                        a.t[o] = t;
                        acc.x += t.x * t.x + t.y * t.y;
                        const double dx = t.x - rv.x, dy = t.y - rv.y;
                        acc.y += dx * dx + dy * dy;
                    }
                }
            });
            gather_sums(ch, acc, Sum{});
        }
        if (!(alive = reduce(Sum{}))) break;
        bool more = false;
        for (int j = tid; j < b; j += NT) {
            const double tn = sqrt(tot[j].x);
            int act = active[j], rst = 0;
            if (accept) {
                // Under the fixed policy a column leaves when the residual of its
                // recurrence meets the threshold.  The true one is some roundings
                // away: at kappa(S) = 50 and a tolerance of 1e-10 by 1e-7 of the
                // threshold, and about one of 10^7 columns misses it; both grow with
                // kappa and with the tightness of the tolerance.  Such a column goes on
                // from its true residual; one that is further off fails.
                rnorm[j] = tn;
                act = rst = !broken && !nonfinite && k < a.maxiter && redos < kMostRedos && tn > thr[j] &&
                            tn <= kRedoWithin * thr[j];
            } else if (act) {
                if (a.adaptive) {
                    const double gap = sqrt(tot[j].y);
                    rst = tn > thr[j] && (gap > a.gap_ratio * fmax(tn, thr[j]) || rnorm[j] <= thr[j]);
                } else {
                    rst = 1;
                }
                act = tn > thr[j];
            }
            active[j] = act;
            restart[j] = rst;
            more |= rst != 0;
        }
        if (accept) {
            if (!__syncthreads_or(more)) break;
            ++redos;
        } else {
            ++checks;
            restarts += __syncthreads_count(more);
        }
        // ---- r <- t on restarted columns, z = M^-1 r
        for (int ch = 0; ch < nch; ++ch) {
            double2 acc = make_double2(0., 0.);
            rows(ch, [&](int li, bool on, int u) {
                if (!on) return;
                const bool rst = restart[u];
                double2 rr[4], zz[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const size_t o = at(ch, li, i);
                    if constexpr (RES) {
                        if (rst) rs[i] = __ldcg(a.t + o);
                        rr[i] = rs[i];
                    } else {
                        rr[i] = rst ? a.t[o] : a.r[o];
                    }
                }
                precondition(li, rr, zz);
                if (first) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const size_t o = at(ch, li, i);
                        a.z[o] = zz[i];
                        if constexpr (!RES) {
                            if (rst) a.r[o] = rr[i];
                        }
                        acc.y += rr[i].x * zz[i].x + rr[i].y * zz[i].y;
                    }
                }
            });
            gather_sums(ch, acc, Sum{});
        }
        if (!(alive = reduce(Sum{}))) break;
        bool left = false;
        for (int j = tid; j < b; j += NT) {
            const double old = rz[j], now = tot[j].y;
            beta[j] = active[j] ? now / (old != 0. ? old : 1.) : 0.;
            rz[j] = now;
            left |= active[j] != 0;
        }
        halt = !__syncthreads_or(left);
    }

    // ---- Y = x safe, with the representability checks (native.cpp:424-444)
    // (only now: Y may be B, which the continuation reads again)
    if (alive) {
        for (int ch = 0; ch < nch; ++ch) {
            double2 acc = make_double2(0., 0.);
            rows(ch, [&](int li, bool on, int u) {
                if (!on || !first || u >= b) return;
                const double sf = safe[u];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    double2 v;
                    if constexpr (RES) v = ys[i];
                    else v = a.y[at(ch, li, i)];
                    const double2 o = make_double2(v.x * sf, v.y * sf);
                    a.Y[(4 * (I0 + li) + i) * (int64_t)b + u] = o;
                    acc.x += (!isfinite(v.x) || !isfinite(v.y)) ? 1. : 0.;
                    acc.y += (!isfinite(o.x) || !isfinite(o.y)) ? 1. : 0.;
                }
            });
            gather_sums(ch, acc, Sum{});
        }
        alive = reduce(Sum{});
    }
    if (blockIdx.x != 0) return;
    // The packets of a solve that gave up may be some numbers ahead.  A CTA that
    // begins after this and reads the new base finds bar[1] set and puts out none,
    // which the next solve would take for its own.
    if (!CL && tid == 0) {
        __threadfence();
        a.bar[2] = seq + (alive ? 0u : 1024u);
    }
    if (!alive) {
        if (tid == 0) atomicOr(a.status + 3, 1);
        return;
    }
    // ---- CTA 0: the per-column report, the counters and the status word
    bool notconv = false, unrep = false;
    for (int j = tid; j < b; j += NT) {
        const int finp = tot[j].x == 0., fin = finp && tot[j].y == 0.;
        const int conv = rnorm[j] <= thr[j] && !brk[j] && fin;
        const double rel = bn[j] > 0. ? rnorm[j] / bn[j] : 0.;
        a.c.conv[j] = conv;
        a.c.brk[j] = brk[j];
        a.c.finp[j] = finp;
        a.c.fino[j] = fin;
        a.c.iters[j] = iters[j];
        a.c.relative[j] = rel;
        a.c.residual[j] = rnorm[j] * safe[j];
        alpha[j] = rel;
        notconv |= !conv;
        unrep |= !fin;
    }
    const bool any_nc = __syncthreads_or(notconv), any_unrep = __syncthreads_or(unrep);
    __shared__ int owns;
    if (tid == 0) {
        int it = 0;
        double rel = a.cnt->max_rel;
        for (int j = 0; j < b; ++j) {
            it = max(it, iters[j]);
            rel = fmax(rel, alpha[j]);
        }
        a.cnt->v[0] += checks;
        a.cnt->v[1] += checks + 1 + redos;
        a.cnt->v[2] += restarts + redos;
        a.cnt->v[3] += it;
        a.cnt->redos += redos;
        a.cnt->max_rel = rel;
        a.c.flags[0] = 1;
        a.c.flags[1] = 0;
        a.c.flags[2] = nonfinite;
        a.c.flags[3] = broken;
        const bool failed = any_nc || broken || nonfinite;
        owns = failed && *a.status == 0;
        if (owns) {
            *a.status = nonfinite ? KMSD_EINVAL : KMSD_EMETRIC;
            a.status[1] = 1;
            if (a.fr != nullptr) {
                a.fr->head.ncols = b;
                a.fr->head.code = *a.status;
                a.fr->head.reason = nonfinite ? 3 : any_unrep ? 2 : broken ? 1 : 0;
            }
        }
    }
    __syncthreads();
    if (owns && a.fr != nullptr)
        for (int j = tid; j < b && j < kMaxReportCols; j += NT) {
            a.fr->converged[j] = (uint8_t)a.c.conv[j];
            a.fr->breakdown[j] = (uint8_t)brk[j];
            a.fr->iterations[j] = iters[j];
            a.fr->true_residual[j] = a.c.residual[j];
            a.fr->relative_residual[j] = a.c.relative[j];
        }
}

enum { kFormCluster = 1, kFormGrid = 2, kFormStream = 3 };
// Smaller systems keep the launch sequence.  Speed does not ask for that: 4 to 63
// block rows of 5 blocks x 1 to 32 columns take 0.46 to 0.59 ms with it and 0.16 to
// 0.20 in one cluster.  A program that reads kmsd_kernel_launches sees its launches
// per iteration, and the tests hold a system of 40 block rows to them.
constexpr int kMinBlockRows = 64;

template <int lcw, bool CPLX>
const void *kernel_form(int form) {
    switch (form) {
        case kFormCluster: return (const void *)pcg_resident_kernel<lcw, CPLX, true, true>;
        case kFormGrid: return (const void *)pcg_resident_kernel<lcw, CPLX, false, true>;
        case kFormStream: return (const void *)pcg_resident_kernel<lcw, CPLX, false, false>;
    }
    return nullptr;
}
constexpr int kMinLcw = 2, kMaxLcw = 5;
const void *kernel_of(int form, int lcw, bool cplx) {
    switch (lcw) {
        case 2: return cplx ? kernel_form<2, true>(form) : kernel_form<2, false>(form);
        case 3: return cplx ? kernel_form<3, true>(form) : kernel_form<3, false>(form);
        case 4: return cplx ? kernel_form<4, true>(form) : kernel_form<4, false>(form);
        case 5: return cplx ? kernel_form<5, true>(form) : kernel_form<5, false>(form);
    }
    return nullptr;
}

// Largest dynamic shared memory of a CTA, and the one-time attributes of the
// kernels.
int smem_limit() {
    static PerDevice<int> limit;
    return limit.get([](int dev) {
        int optin = 0;
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        const int cap = optin - 1024;
        for (int form = kFormCluster; form <= kFormStream; ++form)
            for (int lcw = kMinLcw; lcw <= kMaxLcw; ++lcw)
                for (bool cplx : {false, true}) {
                    const void *k = kernel_of(form, lcw, cplx);
                    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
                    if (form == kFormCluster) cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
                }
        return cap;
    });
}

// Whether 16 CTAs with the largest shared memory fit one cluster on this device.
bool cluster_fits() {
    static PerDevice<bool> fits;
    const int smem = smem_limit();
    return fits.get([smem](int) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(kClusterCtas);
        cfg.blockDim = dim3(kResThreads);
        cfg.dynamicSmemBytes = smem;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = kClusterCtas;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, kernel_of(kFormCluster, kMaxLcw, true), &cfg) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        return n > 0;
    });
}

// Block rows and S blocks of the largest CTA share.
void largest_share(const kmsd_csr_s *S, int ctas, int *own, int *blocks) {
    const int64_t nbr = S->bsr_nb;
    *own = *blocks = 0;
    for (int c = 0; c < ctas; ++c) {
        const int64_t i0 = nbr * c / ctas, i1 = nbr * (c + 1) / ctas;
        *own = std::max(*own, (int)(i1 - i0));
        *blocks = std::max(*blocks, S->bsr_ptr_host[i1] - S->bsr_ptr_host[i0]);
    }
}

// The block columns that each CTA's rows touch (its halo), sorted, with its own
// block rows among them, and every block's place in its CTA's list; nullptr where
// there is no memory for them.
int halo_of(kmsd_metric_s *M, int ctas, kmsd_metric_s::Halo **out) {
    auto it = M->halos.find(ctas);
    if (it != M->halos.end()) {
        *out = &it->second;
        return KMSD_OK;
    }
    const kmsd_csr_s *S = M->S;
    const int64_t nbr = S->bsr_nb, nblk = S->bsr_ptr_host[nbr];
    std::vector<int> off(ctas + 1, 0), list, local(std::max<int64_t>(nblk, 1)), self(nbr), place(nbr);
    kmsd_metric_s::Halo h;
    for (int c = 0; c < ctas; ++c) {
        const int64_t i0 = nbr * c / ctas, i1 = nbr * (c + 1) / ctas;
        const int k0 = S->bsr_ptr_host[i0], k1 = S->bsr_ptr_host[i1];
        std::vector<int> cols(S->bsr_idx_host.begin() + k0, S->bsr_idx_host.begin() + k1);
        for (int64_t i = i0; i < i1; ++i) cols.push_back((int)i);
        std::sort(cols.begin(), cols.end());
        cols.erase(std::unique(cols.begin(), cols.end()), cols.end());
        for (size_t i = 0; i < cols.size(); ++i) place[cols[i]] = (int)i;
        for (int k = k0; k < k1; ++k) local[k] = place[S->bsr_idx_host[k]];
        for (int64_t i = i0; i < i1; ++i) self[i] = place[i];
        list.insert(list.end(), cols.begin(), cols.end());
        off[c + 1] = (int)list.size();
        h.most = std::max(h.most, (int)cols.size());
    }
    const size_t n[4] = {off.size(), list.size(), local.size(), self.size()};
    const std::vector<int> *src[4] = {&off, &list, &local, &self};
    if (h.mem.try_ensure((n[0] + n[1] + n[2] + n[3]) * sizeof(int))) {
        *out = nullptr;
        return KMSD_OK;
    }
    int *d = h.mem.as<int>();
    int **dst[4] = {&h.off, &h.list, &h.local, &h.self};
    for (int i = 0; i < 4; ++i) {
        KMSD_CUDA(cudaMemcpy(d, src[i]->data(), n[i] * sizeof(int), cudaMemcpyHostToDevice));
        *dst[i] = d;
        d += n[i];
    }
    if (settle()) return KMSD_ECUDA;
    auto ins = M->halos.emplace(ctas, h);
    h.mem.p = nullptr;  // owned by the map entry now
    *out = &ins.first->second;
    return KMSD_OK;
}

}  // namespace

namespace kmsd {

int resident_plan(kmsd_metric_s *M, int64_t b, ResidentPlan *out) {
    *out = ResidentPlan{};
    const kmsd_csr_s *S = M->S;
    if (S->bsr_nb < kMinBlockRows || M->nseg > 1 || M->store32) return KMSD_OK;
    if (M->nblocks > 0 && M->ub != 4) return KMSD_OK;
    const bool cplx = S->complex_values;
    const size_t limit = smem_limit();
    const int pre_d = M->nblocks > 0 ? (M->inv_real ? 16 : 32) : 4;
    const int sms = sm_count();
    int full = kMinLcw;  // one chunk for all columns, where 32 are enough
    while ((1 << full) < b && full < kMaxLcw) ++full;
    ResidentPlan pl;
    pl.lcw = full;
    // every thread owns one (block row, column); the blocks of a row are split
    // over as many lanes as are left
    auto resident = [&](int form, int ctas) -> int {
        if ((1 << full) < b || S->bsr_nb > (int64_t)ctas * (kResThreads >> full)) return KMSD_OK;
        largest_share(S, ctas, &pl.own, &pl.blocks);
        if (pl.own > kResThreads >> full) return KMSD_OK;
        auto smem = [&](int most) {
            return state_bytes(kResThreads, 1 << full, form == kFormCluster) +
                   slice_bytes(pl.own, pl.blocks, cplx, pre_d, most, kResidentUnits) + ((size_t)most << (full + 6));
        };
        // a halo holds the CTA's own block rows; its lists are made where it may fit
        if (smem(pl.own) > limit) return KMSD_OK;
        kmsd_metric_s::Halo *h;
        if (int rc = halo_of(M, ctas, &h)) return rc;
        if (!h) return KMSD_OK;
        pl.smem = smem(h->most);
        if (pl.smem > limit) return KMSD_OK;
        pl.form = form;
        pl.ctas = ctas;
        pl.threads = kResThreads;
        pl.lks = 0;
        while (full + pl.lks < 5 && pl.lks < 3 && pl.own <= kResThreads >> (full + pl.lks + 1)) ++pl.lks;
        pl.halo = h;
        return KMSD_OK;
    };
    int rc = KMSD_OK;
    if (cluster_fits()) rc = resident(kFormCluster, kClusterCtas);
    if (!rc && !pl.form) rc = resident(kFormGrid, sms);
    if (rc) return rc;
    if (!pl.form) {
        largest_share(S, sms, &pl.own, &pl.blocks);
        pl.nch = (int)((b + (1 << full) - 1) >> full);
        pl.smem = state_bytes(kStreamThreads, pl.nch << full, false) + slice_bytes(pl.own, pl.blocks, cplx, pre_d, 0, kStreamUnits);
        // A chunk of columns takes the latency of a block row's products whatever the
        // number of rows, and the chunks come one after another, where the launch
        // sequence splits rows and takes all columns at once.  With few rows for each
        // CTA, many chunks and long rows that is slower: 64 / 216 / 512 block rows of
        // 17 blocks x 256 columns took 3.57 / 4.44 / 5.85 ms against 2.36 / 3.63 / 6.34,
        // 64 x 128 2.03 against 2.18, 216 x 192 3.55 against 3.46.  The line fits 672
        // solves of 64 to 900 block rows, 5 to 33 blocks a row and 33 to 256 columns,
        // with at most 14 % lost on either side of it.
        const double row_blocks = (double)S->bsr_ptr_host[S->bsr_nb] / (double)S->bsr_nb;
        const bool slower = pl.nch * (row_blocks + 9.) > 88. + 44. * (double)S->bsr_nb / sms;
        if (pl.smem <= limit && !slower) {
            pl.form = kFormStream;
            pl.ctas = sms;
            pl.threads = kStreamThreads;
            pl.lks = 0;
        }
    }
    if (!pl.form) return KMSD_OK;
    const size_t cols = (size_t)pl.nch << pl.lcw;
    const size_t bytes = 256 + 4 * cols * (pl.ctas + 1) * sizeof(uint4);
    // The vectors are padded to whole chunks, to less than twice b columns from 5 on.
    // Where that does not fit, the launch sequence runs in b columns.
    if ((int64_t)cols >= M->no_room) return KMSD_OK;
    if (M->resident.bytes < bytes) {
        if (M->resident.try_ensure(bytes)) {
            M->no_room = (int64_t)cols;
            return KMSD_OK;
        }
        KMSD_CUDA(cudaMemset(M->resident.p, 0, bytes));
        if (settle()) return KMSD_ECUDA;
    }
    if (M->ensure((int64_t)cols, b)) {
        cudaGetLastError();
        M->no_room = (int64_t)cols;
        for (DevBuf *d : {&M->q, &M->y, &M->r, &M->z, &M->p, &M->sp, &M->t}) d->release();
        return M->ensure(b, b) ? KMSD_ECUDA : KMSD_OK;
    }
    *out = pl;
    return KMSD_OK;
}

int resident_solve(kmsd_metric_s *M, const ResidentPlan &pl, const double2 *B, double2 *Y, int64_t b, double rtol,
                   double atol, int maxiter, cudaStream_t s, int *status, FailReportFull *fr) {
    ResArgs a;
    std::memset(&a, 0, sizeof(a));
    a.S = M->S->bsr64();
    a.b = (int)b;
    a.B = B;
    a.Y = Y;
    a.y = M->y.as<double2>();
    a.r = M->r.as<double2>();
    a.z = M->z.as<double2>();
    a.p = M->p.as<double2>();
    a.sp = M->sp.as<double2>();
    a.t = M->t.as<double2>();
    a.diag = M->diag;
    a.minv = M->nblocks > 0 ? M->factors : nullptr;
    a.minv_real = M->inv_real;
    if (pl.halo) {
        a.halo_off = pl.halo->off;
        a.halo = pl.halo->list;
        a.local = pl.halo->local;
        a.self = pl.halo->self;
        a.halos = pl.halo->most;
    }
    a.c = col_ptr(M->cols.p, b);
    a.cnt = M->dcount.as<Counters>();
    a.rtol = rtol;
    a.atol = atol;
    a.gap_ratio = M->gap_ratio;
    a.maxiter = maxiter;
    a.interval = M->interval;
    a.adaptive = M->adaptive;
    a.status = status;
    a.fr = fr;
    a.bar = M->resident.as<unsigned>();
    a.packets = reinterpret_cast<uint4 *>(M->resident.as<char>() + 256);
    a.lcw = pl.lcw;
    a.lks = pl.lks;
    a.nch = pl.nch;
    a.own = pl.own;
    a.blocks = pl.blocks;
    KMSD_CUDA(cudaMemsetAsync(a.bar, 0, 2 * sizeof(unsigned), s));  // (not the packets' sequence base)
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(pl.ctas);
    cfg.blockDim = dim3(pl.threads);
    cfg.dynamicSmemBytes = pl.smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    if (pl.form == kFormCluster) {
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = pl.ctas;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    } else {
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
    }
    cfg.attrs = at;
    cfg.numAttrs = 1;
    void *args[] = {&a};
    const void *k = kernel_of(pl.form, pl.lcw, a.S.im != nullptr);
    KMSD_CUDA(cudaLaunchKernelExC(&cfg, k, args));
    count_launch();
    return KMSD_OK;
}

}  // namespace kmsd
